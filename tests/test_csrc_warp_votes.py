"""Control flow of warps in the kernels' sources, as far as it can be read off them: a branch that a whole warp takes must not hang on what one lane sees."""
import pathlib
import re

CSRC = pathlib.Path(__file__).parents[1] / "isca-2025-lia_b200" / "csrc"
SOURCES = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*"))}


def test_probes_of_barriers_are_votes():
    """Lanes that probe a barrier one after the other may see it before and after its phase ends, so only a vote may decide where the warp goes."""
    calls = [(name, line.strip()) for name, text in SOURCES.items() for line in text.splitlines() if re.search(r"\bmbar_test\(", line)]
    assert len(calls) >= 2                                          # the probe and the vote
    for name, line in calls:
        assert re.match(r"__device__ __forceinline__ bool mbar_test\(uint32_t bar, uint32_t parity\) \{", line) or "__all_sync(0xffffffffu, mbar_test(" in line, (name, line)
    assert [name for name, text in SOURCES.items() if "mbarrier.test_wait" in text] == ["umma.cuh"]


def test_commits_follow_the_lane_that_issues():
    """A commit follows the products of its own thread alone: where the elected lane issues them, it commits them too, those that are drained after a wait has run out among them."""
    seen = 0
    for name, text in SOURCES.items():
        if not re.search(r"\b(elect_one|mma_\w*if)\(", text) or name == "umma.cuh":
            continue
        for line in text.splitlines():
            seen += "commit_if(" in line
            assert not re.search(r"\btcgen05_commit(_pair)?\(", line) or "if (one)" in line, (name, line.strip())
    assert seen >= 10


def test_rows_that_are_not_put_are_formed_again():
    """Attention's rows whose sums are not finite are left out when rows are written: only where sums are complete, and whoever leaves them out forms them again without a further condition."""
    assert re.search(r"again = __ballot_sync\(0xffffffffu, alive && ", SOURCES["attn_sm100.cuh"])
    callers = [name for name, text in SOURCES.items() if re.search(r"= rows_out\(", text)]
    assert callers == ["latent_attn_sm100.cu", "window_attn_sm100.cu"]
    for name in callers:
        assert re.search(r"rows_out\([^;]*?O, inv, alive, ", SOURCES[name]) and "    if (again) {" in SOURCES[name], name


def test_loads_under_way_are_waited_for_after_the_last_wait():
    """A warp that has asked for all its loads may be done before another's wait runs out: what is under way is waited for behind the block's last barrier, when no wait is left to run out."""
    found = 0
    for name, text in SOURCES.items():
        if "wait_in_flight(" not in text or name == "umma.cuh":
            continue
        last = max(text.rfind(s) for s in ("wait_for(", "warp_wait("))
        assert text.index("wait_in_flight(") > last or name in ("attn_sm100.cuh", "ssd_chunk_sm100.cu"), name      # (one holds functions, the other several kernels without such loads)
        found += "tma_load_2d(" in text
    assert found == 3
