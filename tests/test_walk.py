"""The forward walk (walk.cu) where it can go wrong, against the oracle: paths that are cycles, keys
that tie with the labels of dummy nodes, batches on both sides of its batch-size rules, unaligned
answers, and an index searched with another k than its own."""
import numpy as np
import pytest

import oracle as orc
import sbwt_gpu_b200 as sg
from sbwt_gpu_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _seqs(kind, k, rng):
    g = wl.random_bases(rng, 3000).tobytes().decode()
    if kind == "cycles":  # closed paths: one letter, two letters, a longer period, a circle of the genome
        return ["A" * 80, "CT" * 60, "ACGGT" * 40, g[:700] + g[:700]]
    if kind == "ties":  # keys of A-runs tie with $-padded labels, keys of T-runs with the padding
        return ["A" * (k + 5) + g[:200], "T" * (k + 7), "CA" + "A" * k, g[200:260] + "T" * (k + 1), "AC" * k]
    return [g, g[:1500] + "G" + g[1501:], g[900:1000]]  # "branches"


def _rows(parts):
    starts = np.zeros(len(parts) + 1, dtype=np.uint64)
    starts[1:] = np.cumsum([len(p) for p in parts])
    return np.frombuffer("".join(parts).encode(), dtype=np.uint8), starts


def _search(ix, letters, rows, nk, shift=0):
    import torch
    d_l = torch.from_numpy(letters.copy()).cuda()
    d_r = torch.from_numpy(rows.view(np.int64)).cuda()
    ans = torch.full((nk + 8,), -7, dtype=torch.int64, device="cuda")
    bits = torch.zeros((nk + 31) // 32 + 1, dtype=torch.int32, device="cuda")
    ix.search_reads(d_l, d_r, ans[shift:shift + nk], nk, d_member_bits=bits)
    mem = torch.zeros_like(bits)
    ix.search_reads(d_l, d_r, None, nk, d_member_bits=mem)
    torch.cuda.synchronize()
    a = ans.cpu().numpy()
    assert (a[:shift] == -7).all() and (a[shift + nk:] == -7).all()
    assert torch.equal(bits, mem)
    a = a[shift:shift + nk].view(np.uint64)
    want = np.zeros((nk + 31) // 32 * 32, dtype=np.uint8)
    want[:nk] = a != orc.NOT_FOUND
    got = bits.cpu().numpy().view(np.uint32)[: (nk + 31) // 32]
    assert np.array_equal(got, np.packbits(want, bitorder="little").view(np.uint32))
    return a


@pytest.mark.parametrize("k,p", [(4, 2), (11, 0), (16, 8), (31, 10), (32, 12)])
@pytest.mark.parametrize("kind", ["cycles", "ties", "branches"])
def test_walk_equals_the_oracle(cuda, kind, k, p):
    rng = wl.rng_for(1000 + k)
    seqs = _seqs(kind, k, rng)
    built = sg.build_sbwt([s.encode() for s in seqs], k)
    text = "".join(seqs)
    parts = list(seqs)
    for n in [1, k - 1, k, k + 1, 64, 255, 256, 257, 511, 600]:
        at = int(rng.integers(0, max(1, len(text) - n)))
        read = bytearray(text[at:at + n].encode())
        for i in rng.integers(0, len(read), size=len(read) // 60):
            read[i] = int(wl.ACGT[rng.integers(0, 4)])
        parts += [text[at:at + n], read.decode(), wl.random_bases(rng, n).tobytes().decode(), ""]
    letters, rows = _rows(parts)
    want = orc.OracleIndex(built.bits, built.n_bits).search_reads(letters, rows, k, p)
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        for shift in (0, 1, 3):
            assert np.array_equal(_search(ix, letters, rows, want.size, shift), want)


@pytest.mark.parametrize("reads", [70_000, 70_500])  # below and above the batch that is filled ahead
def test_walk_batch_sizes(cuda, reads):
    rng = wl.rng_for(77)
    k, p = 31, 10
    genome = wl.random_bases(rng, 50_000)
    built = sg.build_sbwt([genome.tobytes()], k)
    letters, rows = wl.mixed_reads(rng, genome, reads // 4, reads - reads // 4, 149, 0.01)
    want = orc.OracleIndex(built.bits, built.n_bits).search_reads(letters, rows, k, p)
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        assert np.array_equal(_search(ix, letters, rows, want.size, 1), want)


@pytest.mark.parametrize("k", [8, 9, 10, 11, 16, 31])  # 8-letter probes: none to all three offsets fall together
@pytest.mark.parametrize("reads", [1_000, 5_000])  # runs of one k-mer, and of several
def test_probes_of_short_and_long_k_mers(cuda, reads, k):
    rng = wl.rng_for(600 + k)
    genome = wl.random_bases(rng, 3_000)
    built = sg.build_sbwt([genome.tobytes()], k)
    letters, rows = wl.mixed_reads(rng, genome, reads // 2, reads - reads // 2, 150, 0.05)
    want = orc.OracleIndex(built.bits, built.n_bits).search_reads(letters, rows, k, 6)
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=6) as ix:
        assert np.array_equal(_search(ix, letters, rows, want.size), want)


@pytest.mark.parametrize("rows", [11_263, 11_264])  # the most rows of the one-launch row table, and one more
@pytest.mark.parametrize("offset", [0, 16, 1])  # alignment of the letters
def test_row_tables(cuda, rows, offset):
    import torch
    rng = wl.rng_for(rows)
    k, p = 21, 8
    genome = wl.random_bases(rng, 30_000)
    built = sg.build_sbwt([genome.tobytes()], k)
    lens = rng.integers(0, 90, size=rows)
    lens[rng.integers(0, rows, size=rows // 3)] = 0
    starts = np.zeros(rows + 1, dtype=np.uint64)
    starts[1:] = np.cumsum(lens)
    letters = np.resize(genome, int(starts[-1])).copy()
    wl.substitute(rng, letters, 0.02)
    want = orc.OracleIndex(built.bits, built.n_bits).search_reads(letters, starts, k, p)
    buf = torch.zeros(letters.size + offset, dtype=torch.uint8, device="cuda")
    buf[offset:] = torch.from_numpy(letters).cuda()
    d_rows = torch.from_numpy(starts.view(np.int64)).cuda()
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        ans = torch.full((want.size + 1,), -7, dtype=torch.int64, device="cuda")
        ix.search_reads(buf[offset:], d_rows, ans, want.size)
        torch.cuda.synchronize()
        got = ans.cpu().numpy().view(np.uint64)
        assert np.array_equal(got[:-1], want) and got[-1] == np.uint64(2**64 - 7)


@pytest.mark.parametrize("dk", [-2, 1])
def test_another_k_than_the_index(cuda, dk):
    """Searched with a k that is not the one of its labels, an index takes the walk without the labels; the
    answers are those of one search per k-mer."""
    rng = wl.rng_for(5)
    k = 21 + dk
    genome = wl.random_bases(rng, 20_000)
    built = sg.build_sbwt([genome.tobytes(), genome[:500].tobytes()], 21)
    letters, rows = wl.mixed_reads(rng, genome, 60, 60, 150, 0.01)
    nk = sg.count_kmers(rows, k)
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=8) as ix:
        got = _search(ix, letters, rows, nk)
        ix.set_search_mode(sg.SEARCH_EVERY_KMER)
        assert np.array_equal(got, _search(ix, letters, rows, nk))


@pytest.mark.parametrize("k,p", [(4, 2), (16, 8), (31, 10), (32, 12)])
def test_kmer_lists_equal_the_oracle(cuda, k, p):
    """Lists of single k-mers on both sides of a warp's and a block's share, and positions without runs."""
    import torch
    rng = wl.rng_for(2000 + k)
    seqs = _seqs("ties", k, rng) + _seqs("branches", k, rng)
    built = sg.build_sbwt([s.encode() for s in seqs], k)
    text = "".join(seqs)
    at = rng.integers(0, len(text) - k + 1, size=3000)
    parts = [text[i:i + k] for i in at]
    parts[::3] = [wl.random_bases(rng, k).tobytes().decode() for _ in parts[::3]]
    letters, rows = _rows(parts)
    want = orc.OracleIndex(built.bits, built.n_bits).search_reads(letters, rows, k, p)
    codes = np.searchsorted(wl.ACGT, letters).reshape(-1, k).astype(np.uint64)
    words = np.zeros(len(parts), dtype=np.uint64)
    for i in range(k):
        words |= codes[:, i] << np.uint64(62 - 2 * i)
    junk = rng.integers(0, 2**63, size=words.size, dtype=np.int64).astype(np.uint64)
    if k < 32:
        words |= junk & np.uint64((1 << (64 - 2 * k)) - 1)  # letters past the k-mer do not count
    d_words = torch.from_numpy(words.view(np.int64)).cuda()
    packed = torch.from_numpy(wl.pack_words(np.frombuffer((text + "A" * 32).encode(), dtype=np.uint8)).view(np.int64)).cuda()
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        for n in (1, 31, 32, 33, 127, 128, 129, 511, 513, 3000):
            ans = torch.full((n + 1,), -7, dtype=torch.int64, device="cuda")
            ix.search_kmers(d_words, ans, n)
            torch.cuda.synchronize()
            got = ans.cpu().numpy().view(np.uint64)
            assert np.array_equal(got[:n], want[:n]) and got[n] == np.uint64(2**64 - 7)
        pos = torch.from_numpy(at.astype(np.int64)).cuda()  # random positions: no runs
        ix.search_packed(packed, pos, pos.numel())
        torch.cuda.synchronize()
        l2, r2 = _rows([text[i:i + k] for i in at])
        want2 = orc.OracleIndex(built.bits, built.n_bits).search_reads(l2, r2, k, p)
        assert np.array_equal(pos.cpu().numpy().view(np.uint64), want2)


def test_membership_only_with_full_pools(cuda):
    """Membership alone, with runs that go back to be probed while others are taken from the same pool: reads of
    which every tenth letter or so is substituted, so that each run changes hands many times."""
    import torch
    rng = wl.rng_for(4100)
    k, p = 21, 8
    genome = wl.random_bases(rng, 40_000)
    built = sg.build_sbwt([genome.tobytes()], k)
    ox = orc.OracleIndex(built.bits, built.n_bits)
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        for length, sub in ((280, 0.01), (280, 0.1), (60, 0.03)):
            letters, rows = wl.mixed_reads(rng, genome, 20_000, 500, length, sub)
            want = ox.search_reads(letters, rows, k, p) != orc.NOT_FOUND
            d_l, d_r = torch.from_numpy(letters).cuda(), torch.from_numpy(rows.view(np.int64)).cuda()
            for _ in range(3):
                bits = torch.full(((want.size + 31) // 32,), -1, dtype=torch.int32, device="cuda")
                ix.search_reads(d_l, d_r, None, want.size, d_member_bits=bits)
                got = np.unpackbits(bits.cpu().numpy().view(np.uint8), bitorder="little")
                assert np.array_equal(got[:want.size].astype(bool), want) and not got[want.size:].any()


def test_graph_replay_after_the_kernel_contract(cuda):
    """The kernel contract grows scratch that a captured search of reads uses: the next search captures again."""
    import torch
    rng = wl.rng_for(4200)
    k, p = 31, 10
    genome = wl.random_bases(rng, 40_000)
    built = sg.build_sbwt([genome.tobytes()], k)
    letters, rows = wl.mixed_reads(rng, genome, 6_000, 6_000, 60, 0.01)  # more rows than one launch prepares
    ox = orc.OracleIndex(built.bits, built.n_bits)
    want = ox.search_reads(letters, rows, k, p)
    words = torch.from_numpy(wl.pack_words(genome).view(np.int64)).cuda()
    s = torch.cuda.Stream()
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        ix.use_graphs(True)
        d_l, d_r = torch.from_numpy(letters).cuda(), torch.from_numpy(rows.view(np.int64)).cuda()
        ans = torch.empty(want.size, dtype=torch.int64, device="cuda")
        for contract in (0, 30_000, 39_000):
            if contract:
                pos = torch.arange(contract, dtype=torch.int64, device="cuda")
                torch.cuda.synchronize()
                ix.search_packed(words, pos, stream=s)
                s.synchronize()
                ref = ox.search_reads(genome[:contract + k - 1], np.array([0, contract + k - 1], dtype=np.uint64), k, p)
                assert np.array_equal(pos.cpu().numpy().view(np.uint64), ref)
            ans.fill_(-7)
            torch.cuda.synchronize()
            ix.search_reads(d_l, d_r, ans, want.size, stream=s)
            s.synchronize()
            assert np.array_equal(ans.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("layout", [sg.SBWT_LAYOUT_LINES, sg.SBWT_LAYOUT_POPPY])
def test_autotune_tries_what_the_walk_reads(cuda, layout):
    """The forward walk is the same on every layout: the tuner leaves the lines, times the others with kernels that
    read them, tries no table that the walk does not read, and the reads behind the prefilter still run."""
    import torch
    rng = wl.rng_for(4300)
    k, p = 31, 8
    genome = wl.random_bases(rng, 30_000)
    built = sg.build_sbwt([genome.tobytes()], k)
    letters, rows = wl.mixed_reads(rng, genome, 200, 200, 150, 0.01)
    want = orc.OracleIndex(built.bits, built.n_bits).search_reads(letters, rows, k, p)
    d_l, d_r = torch.from_numpy(letters).cuda(), torch.from_numpy(rows.view(np.int64)).cuda()
    ans = torch.empty(want.size, dtype=torch.int64, device="cuda")
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        ix.configure(layout)
        rep = ix.autotune(d_l, d_r, ans, want.size, tune_poppy=True)
        cands = rep["candidates"]
        assert rep["best"]["layout"] == "lines" and rep["best"]["mode"] == "stream"
        assert {c["layout"] for c in cands if c["mode"] == "skip"} == {"lines512", "lines2048", "poppy"}
        assert all(c["layout"] == "lines" for c in cands[1:] if c["mode"] == "stream")
        assert len({c["compact_presearch"] for c in cands}) == 1
        with sg.Prefilter.train(ix, steps=20, batch=256, n_positive=2_000, n_negative=2_000) as pf:
            ans.fill_(-7)
            ix.search_reads_filtered(pf, d_l, d_r, ans, want.size)
            torch.cuda.synchronize()
            assert np.array_equal(ans.cpu().numpy().view(np.uint64), want)
        ix.set_search_mode(sg.SEARCH_SKIP_ABSENT)  # the layouts differ: any may be left
        rep = ix.autotune(d_l, d_r, ans, want.size, tune_poppy=True)
        assert {c["mode"] for c in rep["candidates"]} == {"skip"}
        assert len({c["compact_presearch"] for c in rep["candidates"]}) == 2
        torch.cuda.synchronize()
        assert np.array_equal(ans.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("layout", [sg.SBWT_LAYOUT_LINES, sg.SBWT_LAYOUT_LINES512, sg.SBWT_LAYOUT_POPPY])
def test_the_l2_window_covers_the_lines_that_the_walk_reads(cuda, layout):
    import torch
    from cuda.bindings import runtime as rt
    rng = wl.rng_for(4400)
    k, p = 31, 8
    genome = wl.random_bases(rng, 30_000)
    built = sg.build_sbwt([genome.tobytes()], k)
    letters, rows = wl.mixed_reads(rng, genome, 50, 50, 150, 0.01)
    nk = sg.count_kmers(rows, k)
    d_l, d_r = torch.from_numpy(letters).cuda(), torch.from_numpy(rows.view(np.int64)).cuda()
    ans = torch.empty(nk, dtype=torch.int64, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        ix.configure(layout)
        ix.set_walk_options(l2_persist=1)
        ix.search_reads(d_l, d_r, ans, nk, stream=s)  # takes the set-aside and the workspace
        s.synchronize()
        assert rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == 0
        ix.search_reads(d_l, d_r, ans, nk, stream=s)
        err, graph = rt.cudaStreamEndCapture(s.cuda_stream)
        assert err == 0
        count = rt.cudaGraphGetNodes(graph)[-1]
        windows = []
        for node in rt.cudaGraphGetNodes(graph, count)[1]:
            if rt.cudaGraphNodeGetType(node)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel:
                err, val = rt.cudaGraphKernelNodeGetAttribute(
                    node, rt.cudaLaunchAttributeID.cudaLaunchAttributeAccessPolicyWindow)
                assert err == 0
                windows.append(int(val.accessPolicyWindow.num_bytes))
        rt.cudaGraphDestroy(graph)
    lines = (built.n_bits // 224 + 1 + 7) // 8 * 8
    assert max(windows) == 4 * lines * 32


@pytest.mark.parametrize("order", ["reads", "shuffled"])
def test_kernel_contract_of_a_batch_that_is_filled_ahead(cuda, order):
    """From 8M k-mers on the absent answers are written before the walk, over the caller's positions: only where the
    walk takes the call.  Shuffled, the positions form no runs and the list search still has to find them there.  The
    answers start off the 32-byte stores' alignment."""
    import torch
    rng = wl.rng_for(4500)
    k, p, reads, length = 31, 10, 71_000, 149
    genome = wl.random_bases(rng, 50_000)
    built = sg.build_sbwt([genome.tobytes()], k)
    letters, rows = wl.mixed_reads(rng, genome, reads // 4, reads - reads // 4, length, 0.01)
    want = orc.OracleIndex(built.bits, built.n_bits).search_reads(letters, rows, k, p)
    assert want.size > 8 << 20
    per = length - k + 1
    pos = (np.arange(reads, dtype=np.int64)[:, None] * length + np.arange(per)).reshape(-1)
    if order == "shuffled":
        at = rng.permutation(pos.size)
        pos, want = pos[at], want[at]
    words = torch.from_numpy(wl.pack_words(letters).view(np.int64)).cuda()
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        buf = torch.full((pos.size + 4,), -7, dtype=torch.int64, device="cuda")
        buf[1:1 + pos.size] = torch.from_numpy(pos).cuda()
        ix.search_packed(words, buf[1:1 + pos.size], pos.size)
        torch.cuda.synchronize()
        got = buf.cpu().numpy().view(np.uint64)
        assert np.array_equal(got[1:1 + pos.size], want)
        assert (got[:1] == np.uint64(2**64 - 7)).all() and (got[1 + pos.size:] == np.uint64(2**64 - 7)).all()


@pytest.mark.parametrize("kind,dk,walks", [("plain", -2, True), ("plain", 1, True), ("variants", -2, False),
                                           ("variants", -1, False), ("variants", 1, True), ("variants", 3, True)])
def test_which_walk_another_k_takes(cuda, kind, dk, walks):
    """A smaller k than the index's makes labels equal where sequences differ only in the letters that it drops: the
    check of the structures finds them and the right-to-left walk searches.  A larger one, or a smaller one that makes
    none equal, leaves the structures consistent, and the forward walk searches, with the same answers.  (A small
    batch takes a few blocks of the forward walk; the other one's grid fills the device.)"""
    import torch
    rng = wl.rng_for(4600)
    k = 21 + dk
    genome = wl.random_bases(rng, 8_000)
    seqs = [genome.tobytes()]
    if kind == "variants":
        for _ in range(3):
            var = genome.copy()
            wl.substitute(rng, var, 0.02)
            seqs.append(var.tobytes())
    built = sg.build_sbwt(seqs, 21)
    parts = [s[at:at + 90].decode() for s in seqs for at in rng.integers(0, 7_900, size=24 // len(seqs))]
    letters, rows = _rows(parts + [wl.random_bases(rng, 90).tobytes().decode() for _ in range(4)])
    want = orc.OracleIndex(built.bits, built.n_bits).search_reads(letters, rows, k, 8)
    assert 0.3 < (want != orc.NOT_FOUND).mean() < 0.95
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=8) as ix:
        assert np.array_equal(_search(ix, letters, rows, want.size), want)
        ix.profile(True)
        ans = torch.empty(want.size, dtype=torch.int64, device="cuda")
        ix.search_reads(torch.from_numpy(letters.copy()).cuda(), torch.from_numpy(rows.view(np.int64)).cuda(), ans, want.size)
        torch.cuda.synchronize()
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        assert (ix.last_profile()["search_blocks"] < sms) == walks
