"""The rank structures behind the search modes that rank in them.

The default mode walks the paths of the graph on the 32-byte lines whatever the layout, so the poppy and
wide-line rankers are reached only with the absent-run skip and with every k-mer searched: each (superblock, kind)
pair and each wide layout here in both, against the oracle, and the reference program's own output through the
command line on the poppy layout."""
import gzip
import os
import subprocess

import numpy as np
import pytest

import oracle as orc
import sbwt_gpu_b200 as sg
from sbwt_gpu_b200 import workloads as wl

pytestmark = pytest.mark.gpu

CASES = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "cases")


@pytest.fixture(scope="module")
def small(cuda):
    rng = wl.rng_for(4242)
    k, p = 31, 8
    genome = wl.random_bases(rng, 120_000)
    built = sg.build_sbwt([genome.tobytes()], k)
    letters, rows = wl.mixed_reads(rng, genome, 300, 300, 150, 0.01)
    want = orc.OracleIndex(built.bits, built.n_bits).search_reads(letters, rows, k, p)
    with sg.Index.from_bits(built.bits, built.n_bits, k=k, k_presearch=p) as ix:
        yield {"ix": ix, "letters": letters, "rows": rows, "want": want}


def _check(small):
    import torch
    ix, want = small["ix"], small["want"]
    d_l = torch.from_numpy(small["letters"]).cuda()
    d_r = torch.from_numpy(small["rows"].view(np.int64)).cuda()
    for mode in (sg.SEARCH_SKIP_ABSENT, sg.SEARCH_EVERY_KMER):
        ix.set_search_mode(mode)
        ans = torch.full((want.size,), -7, dtype=torch.int64, device="cuda")
        bits = torch.zeros((want.size + 31) // 32, dtype=torch.int32, device="cuda")
        ix.search_reads(d_l, d_r, ans, want.size, d_member_bits=bits)
        torch.cuda.synchronize()
        assert np.array_equal(ans.cpu().numpy().view(np.uint64), want), mode
        got = np.unpackbits(bits.cpu().numpy().view(np.uint8), bitorder="little")[: want.size]
        assert np.array_equal(got.astype(bool), want != orc.NOT_FOUND), mode


@pytest.mark.parametrize("sb,kind", orc.SB_KINDS)
def test_queue_fed_search_ranks_in_poppy(small, sb, kind):
    small["ix"].configure(sg.SBWT_LAYOUT_POPPY, bits_in_superblock=sb, rank_structure=kind, kmers_per_thread=0)
    _check(small)


@pytest.mark.parametrize("layout", [sg.SBWT_LAYOUT_LINES, sg.SBWT_LAYOUT_LINES512, sg.SBWT_LAYOUT_LINES2048])
def test_queue_fed_search_ranks_in_the_lines(small, layout):
    small["ix"].configure(layout, kmers_per_thread=0)
    _check(small)


@pytest.mark.parametrize("mode", ["skip", "every"])
@pytest.mark.parametrize("case", sorted(c for c in os.listdir(CASES)
                                        if os.path.exists(os.path.join(CASES, c, "reference.out.gz"))))
def test_cli_on_poppy_matches_reference_program(cuda, case, mode):
    import make_golden
    want = gzip.open(os.path.join(CASES, case, "reference.out.gz")).read()
    r = subprocess.run([sg.CLI_PATH] + make_golden.case_flags(case, CASES) + ["--layout=poppy", f"--search-mode={mode}"],
                       capture_output=True, timeout=300)
    assert r.returncode == 0, r.stderr.decode()
    assert r.stdout == want
