"""Memory ordering inside a warp, read from the kernels' sources (a race shows no fault on a
run that happens to be in step).  Votes and shuffles order no memory: what one lane stores
and another reads has a __syncwarp between."""
import os
import re

import pytest

from conftest import PKG


def source(name):
    """The file's text without comments."""
    with open(os.path.join(PKG, "csrc", name)) as f:
        return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", f.read(), flags=re.S))


def kernel(name, function):
    """The body of a __global__ function."""
    text = source(name)
    head = re.search(r"__global__[^;{]*?\b" + function + r"\(", text)
    start = text.index("{", head.end())
    depth = 0
    for k in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[start:k + 1]
    raise AssertionError(function)


CELL_KERNELS = [("sadmc_cell_kernel.cuh", "cell_move_kernel"), ("sadmc_cell.cu", "wca_grand_kernel")]


@pytest.mark.parametrize("name,function", CELL_KERNELS)
def test_proposal_is_stored_before_it_is_read(name, function):
    """Three lanes of a group store the proposal, an axis each; all of them read it."""
    body = kernel(name, function)
    stores = [m.end() for m in re.finditer(r"\bP\.\w+(\[\w+\])+\s*=[^=]", body)]
    reads = [m.start() for m in re.finditer(r"\(P\.\w+|= P\.\w+", body) if m.start() > max(stores)]
    assert stores and reads
    assert "__syncwarp()" in body[max(stores):min(reads)]


@pytest.mark.parametrize("name,function", [("sadmc_grand.cu", "lj_grand_kernel"), ("sadmc_cell.cu", "wca_grand_kernel")])
def test_proposed_bin_is_read_before_it_is_stored(name, function):
    """Every lane of a group reads the proposed bin's fields (and the bucket's word) to decide;
    one lane of it then books the move in them."""
    body = kernel(name, function)
    decide, book = body.index("bk.lean_decide("), body.index("bk.lean_finish(")
    assert decide < book
    assert "__syncwarp()" in body[decide:book]


SPREAD_KERNELS = [("sadmc_lj_kernel.cuh", "lj_descent_kernel"), ("sadmc_lj_kernel.cuh", "lj_move_kernel"),
                  ("sadmc_lj_lane.cu", "lj_lane_kernel"), ("sadmc_ising.cu", "ising_move_kernel"),
                  ("sadmc_cell_kernel.cuh", "cell_descent_kernel"), ("sadmc_cell_kernel.cuh", "cell_move_kernel"),
                  ("sadmc_grand.cu", "lj_grand_kernel"), ("sadmc_cell.cu", "wca_grand_kernel")]


@pytest.mark.parametrize("name,function", SPREAD_KERNELS)
def test_one_lane_group_to_a_walker(name, function):
    """A lane group without a walker of its own must not run another group's walker: that one
    stores to the planes, spins and lists which the copy would read, with nothing between."""
    body = kernel(name, function)
    assert re.search(r"\bw = warp \* wpw \+ group;", body)
    assert "n_walkers - 1" not in body
    load = re.search(r"\w\.load\(m|= m\.cores\[w\]", body).start()
    assert re.search(r"if \(group >= wpw \|\| w >= m\.n_walkers\) return;", body[:load]) or re.search(
        r"own = group < wpw && w < m\.n_walkers;.*if \(\(TRIAL \|\| m\.descent\) && !own\) return;.*if \(TRIAL \|\| own\) f$", body[:load], re.S)


@pytest.mark.parametrize("name", ["sadmc_fh.cuh", "sadmc_grand_book.cuh"])
def test_one_lane_counts_in_memory(name):
    """A read-modify-write of a plane by all lanes of a group counts once only if they stay in
    step."""
    text = source(name)
    steps = [m for m in re.finditer(r"\b(rt|wlh|tr_att|tr_acc)\[(?:[^\[\]]|\[\w+\])+\] (\+= 1|= \1\[)", text)]
    assert steps
    for m in steps:
        assert re.search(r"if \((leads\(\)|lead)\) (\{[^}]*)?$", text[:m.start()]), m.group()


def test_stage_count_is_read_before_it_is_stored():
    """The general path's Wang-Landau update: every lane reads the bin's stage count, and stores
    the next one."""
    update = source("sadmc_fh.cuh").split("void wl_update()")[1].split("void wl_count(")[0]
    read, count = update.rindex("wlh[k]"), update.rindex("wl_count(")
    assert "sync();" in update[read:count]


@pytest.mark.parametrize("name,function", [
    ("sadmc_lj_kernel.cuh", "lj_move_kernel"), ("sadmc_lj_lane.cu", "lj_lane_kernel"), ("sadmc_ising.cu", "ising_move_kernel"),
    ("sadmc_cell_kernel.cuh", "cell_move_kernel"), ("sadmc_da_kernel.cuh", "lj_da_kernel")])
def test_lean_decision_reads_before_the_booking_stores(name, function):
    """The lean decision reads the proposed bin's stamp and stage count on every lane; the
    booking stores them (the general path's likewise, inside decide_de)."""
    body = kernel(name, function)
    decide, book = re.search(r"fh\.lean_(decide|delayed)\(", body).start(), body.index("fh.decide_de(")
    assert decide < book and re.search(r"__syncwarp\(\);.*if \(SADMC_RARE\(r == 2\)\)", body[decide:book], re.S)
    general = source("sadmc_fh.cuh").split("bool decide_de(")[1].split("bool rejects(")[0]
    assert "sync();" in general[general.index("rejects("):]
