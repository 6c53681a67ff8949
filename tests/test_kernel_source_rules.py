"""Rules that the CUDA sources keep and that no run can show: a breach is a race or a hang that almost never happens."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flat-attention_b200", "csrc")


def functions(text):
    """name -> (header, body) of every function that runs on the device."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
    found = {}
    for m in re.finditer(r"(?:__global__|__device__)[^;{}()]*?\b(\w+)\s*\(", text):
        at, depth = m.end(), 1
        while depth:  # the parameter list
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        rest = re.match(r"\s*(?:const)?\s*\{", text[at:])
        if not rest:
            continue
        start = end = at + rest.end()
        depth = 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        header, body = found.get(m.group(1), ("", ""))  # overloads and specialisations count as one
        found[m.group(1)] = (header + text[m.start():start], body + text[start:end])
    return found


def sources():
    shared = "".join(open(f).read() for f in sorted(glob.glob(os.path.join(CSRC, "*.cuh"))))
    return {os.path.basename(f): functions(open(f).read() + shared) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")))}


def reached(found, kernel):
    """The kernel and every device function of the file that it calls."""
    seen, todo = set(), [kernel]
    while todo:
        name = todo.pop()
        if name not in seen:
            seen.add(name)
            todo += [n for n in found if re.search(r"\b%s\s*(?:<[^;(){}]*>)?\s*\(" % n, found[name][1])]
    return seen


KERNELS = [(f, k) for f, found in sources().items() for k, (header, body) in found.items()
           if "__global__" in header and "grid_dependency_wait" in body]


def test_the_dependent_kernels_are_found():
    assert {k for _, k in KERNELS} >= {"decode_cluster_kernel", "decode_mma_kernel", "merge_row_kernel", "fwd_sm100_kernel", "fwd_f32_kernel",
                                       "fwd_split_merge_kernel", "rotate_to_f16_kernel", "bwd_prep_kernel", "bwd_sm100_kernel"}


@pytest.mark.parametrize("file,kernel", KERNELS)
def test_dependent_kernels_do_not_read_through_the_read_only_path(file, kernel):
    """A kernel that may start while the one before it still writes what it reads must not promise the hardware that this memory
    does not change: no ld.global.nc, no __ldg, and no pointer that lets the compiler choose them."""
    found = sources()[file]
    for name in reached(found, kernel):
        header, body = found[name]
        assert not re.search(r"\.nc\b|__ldg\s*\(", body), name
        assert not re.search(r"const\s+[\w:]+\s*\*\s*__restrict__", header), name


# bwd_sm100_kernel is never the last of its call: its dependent is the dQ kernel, which waits before it touches memory
@pytest.mark.parametrize("file,kernel", [x for x in KERNELS if x[1] != "bwd_sm100_kernel"])
def test_the_last_kernel_of_a_call_lets_its_dependent_start_behind_its_own_wait(file, kernel):
    """The dependent may be the application's: what it does before it waits may count on everything before this kernel.  (The
    forward behind its K rotation does not wait first: the rotation lets nothing start before its blocks, which wait, have ended.)"""
    body = sources()[file][kernel][1]
    for launch in re.finditer(r"grid_dependency_launch\(\)", body):
        assert re.search(r"grid_dependency_wait\(\);\s*$", body[:launch.start()]), body[:launch.start()][-200:]
    if kernel == "rotate_to_f16_kernel":
        assert "grid_dependency_launch" not in body


def enclosing_conditions(body, at):
    """The text in front of each block that is open at position `at`, outermost first."""
    stack, last = [], 0
    for i, ch in enumerate(body[:at]):
        if ch == "{":
            stack.append(body[last:i])
        elif ch == "}":
            stack.pop()
        if ch in "{};":
            last = i + 1
    return stack


@pytest.mark.parametrize("file,kernel", [("fwd_sm100.cu", "fwd_sm100_kernel"), ("bwd_sm100.cu", "bwd_sm100_kernel"),
                                         ("bwd_sm100.cu", "bwd_dq_sm100_kernel"), ("bwd_sm100.cu", "bwd_dq_spill_kernel")])
def test_warps_leave_a_wait_that_gave_up_as_a_whole(file, kernel):
    """mbar_wait answers each lane for itself; warps whose lanes all wait take mbar_wait_warp, which answers them alike."""
    body = sources()[file][kernel][1]
    calls = list(re.finditer(r"\bmbar_(?:wait|wait_warp)\(", body))
    assert calls
    for call in calls:
        one_thread = any("elect_one()" in condition for condition in enclosing_conditions(body, call.start()))
        assert one_thread == (call.group() == "mbar_wait("), body[call.start() - 80:call.end() + 60]


def test_the_warp_wide_wait_answers_every_lane_alike():
    body = sources()["fwd_sm100.cu"]["mbar_wait_warp"][1]  # for one phase and for two
    answers = re.findall(r"return([^;]*);", body)
    assert answers
    for answer in answers:
        votes = answer.split("||")
        assert all(vote.strip().startswith("__all_sync(0xffffffffu,") for vote in votes)
