"""CPU checks of rules that the kernels' source has to keep and that no run can show (a memory-model race that the hardware's
in-order issue hides, a figure in a comment that a layout constant contradicts)."""
import os
import re

import lightop_b200

CSRC = os.path.join(os.path.dirname(lightop_b200.__file__), "csrc")


def _statements(name):
    """The file's statements in order, comments removed and white space folded."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    return [re.sub(r"\s+", " ", s).strip() for s in re.split(r"[;{}]", text) if s.strip()]


def test_an_arrive_orders_the_reads_of_the_whole_warp():
    # what a barrier hands back was read by all lanes of a warp: either every lane arrives for itself, or lane 0 does behind a
    # __syncwarp() (neither converged execution nor a vote orders memory)
    st = _statements("grouped_gemm.cu")
    one = [i for i, s in enumerate(st) if re.match(r"if \(lane == 0\) mbar_arrive(_addr)?\(", s)]
    assert len(one) >= 5
    bare = [f"{st[i - 1]}; {st[i]}" for i in one if st[i - 1] != "__syncwarp()"]
    assert not bare, bare
    # the partial buffers: the one barrier that every lane arrives at, and counted so
    assert "mbar_arrive_addr(used)" in st and "mbar_init(&sm.consumed[s], EPI_WARPS * 32)" in st


def test_what_one_lane_waited_for_is_ordered_before_the_mma():
    # the MMA issuer's two polling lanes agree by a vote; the elected lane issues only after a __syncwarp() that follows it
    st = _statements("grouped_gemm.cu")
    wait = next(i for i, s in enumerate(st) if "LO_SLEEP_MMA)" in s and s.startswith("seen = "))
    issue = next(i for i, s in enumerate(st) if i > wait and "elect_one()" in s)
    vote = max(i for i in range(wait, issue) if "__all_sync" in st[i])
    assert "__syncwarp()" in st[vote + 1:issue]


def test_vector_stores_to_the_callers_output_look_at_its_address():
    # the 16-byte row stores are decided on the host from the row length and the address, not from the length alone
    st = _statements("grouped_gemm.cu")
    assert any(s.startswith("p.vec_store = ") and "& 7) == 0" in s and "a.C) & 15) == 0" in s for s in st)
    i = next(i for i, s in enumerate(st) if "*reinterpret_cast<uint4 *>(dst) = v" in s)
    assert st[i - 1] == "if (p.vec_store)"


def test_silu_quantiser_loads_no_row_that_does_not_exist():
    # the grid is the capacity (with an expert map mostly rows that do not exist): both counts are looked at before a load of the row
    st = _statements("quant.cu")
    first_load = next(i for i, s in enumerate(st) if s == "gv[v] = g[i]")
    assert any(s.startswith("if (num_rows_dev && row >= *num_rows_dev) return") for s in st[:first_load])
    assert any(s.startswith("if (group_counts && row % group_rows >= group_counts[row / group_rows]) return") for s in st[:first_load])


def test_lanes_without_a_group_take_no_quotient():
    # they join the group's maximum and return before the first division (theirs would be the slowest one of the warp)
    st = _statements("quant.cu")
    start = next(i for i, s in enumerate(st) if "float quantise" in s)
    leave = next(i for i in range(start, len(st)) if st[i].startswith("if (!active) return"))
    assert any("__shfl_xor_sync" in s for s in st[start:leave])
    assert not any("__fdiv_rn" in s or "div_by" in s for s in st[start:leave])


def test_what_lets_the_next_kernel_start_has_waited_itself():
    # a kernel that released its successor before its own wait would let it (and what that one releases) run ahead of earlier work
    import glob
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        st = _statements(os.path.basename(path))
        waited = False
        for s in st:
            if "__global__" in s:
                waited = False
            if s.endswith("dependency_wait()"):
                waited = True
            elif s.endswith("dependency_release()"):
                assert waited, os.path.basename(path)
                seen += 1
    assert seen >= 9


def test_the_linear_of_a_few_rows_has_the_ctas_its_rules_count_with():
    # outputs a CTA and the limit on the outputs assume ROW_CTAS CTAs a SM: the compiler has to be held to it wherever a call has more CTAs than
    # there are SMs (a second wave repeats the quantisation)
    with open(os.path.join(CSRC, "quant.cu")) as f:
        text = f.read()
    assert re.search(r"__launch_bounds__\(ROW_THREADS, CTAS\) linear_rows_kernel", text)
    forms = re.findall(r"^(.*)\bLO_ROWS_CASE\((\w+), (\w+)\);", text, flags=re.M)
    assert len(forms) == 4
    for before, _, ctas in forms:
        assert ctas == "ROW_CTAS" or "(int)grid.x <= sm_count()" in before
    assert "ctas = (int64_t)ROW_CTAS * sm_count()" in text and "N > outs * ctas" in text and "N > (int64_t)ROW_OUTS_MAX * ROW_CTAS * sm_count()" in text


def test_every_commit_has_arrived_before_a_cta_leaves():
    # per channel nobody but the weight producer waits for the commits of the steps, and it waits NW steps late: behind its loop it waits for the
    # last NW, in each CTA of a pair (the closing barrier of a cluster orders threads, not arrivals still on their way)
    st = _statements("grouped_gemm.cu")
    loop = next(i for i, s in enumerate(st) if s.startswith("tma_load_2d(sm.w[s]"))
    end = next(i for i in range(loop, len(st)) if "warp == 3" in st[i])
    tail = " ; ".join(st[loop:end])
    assert "if constexpr (MODE == GEMM_CHANNEL)" in tail
    assert "u = it < (uint32_t)NW ? 0u : it - NW" in tail and "ok = mbar_wait(sm, &sm.done[u % ND], (u / ND) & 1u," in tail
