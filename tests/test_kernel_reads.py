"""Kernels that may start before their predecessor has ended (they begin with
after_predecessor()) read what a sort writes by ordinary loads only.  The
read-only path (__ldg, and const pointers declared __restrict__, which let the
compiler choose it) is for data that nobody writes while the kernel runs; such
a load may also be moved above the wait.  The arena and the offsets are such
data, the lists and tables of a round are not.  Checked in the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "string-sorting_b200", "csrc")
# Of the kernels that do wait, and of the functions they share: inputs of the
# sort only.  `jobs`, `text`: used by ordinary launches only.
INPUTS = {"arena", "offs", "jobs", "text"}


def functions():
    """(name, head, body) of the file's functions."""
    with open(os.path.join(CSRC, "ssort_kernels.cu")) as f:
        src = re.sub(r"//[^\n]*|__launch_bounds__\([^)]*\)", "", f.read())
    for m in re.finditer(r"^(?:template[^\n]*\n)?(__global__|__device__)[^;{]*?"
                         r"(\w+)\(([^;{]*?)\)\s*\{", src, re.M):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        yield m.group(2), m.group(0), src[m.end():i]


def test_reads_of_a_sorts_own_data_take_no_read_only_path():
    seen, bad = set(), []
    for name, head, body in functions():
        waits = "after_predecessor();" in body
        if waits:
            seen.add(name)
        if "__global__" in head and not waits:
            continue  # an ordinary launch: its predecessor has ended
        for ptr in re.findall(r"const \w+ \*__restrict__ (\w+)", head + body):
            if ptr not in INPUTS:
                bad.append(f"{name}: {ptr}")
        if "__ldg(" in body and name not in ("load_key", "string_offset", "gather_keys_at"):
            bad.append(f"{name}: __ldg")
    assert {"k_sample", "k_count", "k_scatter", "k_emit", "k_round_end", "k_warp1", "k_equal",
            "k_segsort", "k_segsort_class", "k_warpsort", "k_gather", "k_seg_tiles",
            "k_scan_lookback"} <= seen
    assert not bad, bad
