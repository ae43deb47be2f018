"""Rules of the kernels that no run can show broken: a violation works on the
hardware at hand or depends on how a warp happens to be scheduled, so the
sources are looked at instead."""
import os
import re

from conftest import ROOT


def body(path, start):
    """Source of the function whose definition contains `start`, without comments."""
    src = open(os.path.join(ROOT, "plant_gb300", "csrc", path)).read()
    src = re.sub(r"//[^\n]*", "", src)
    at = src.index(start)
    i = src.index("{", src.index(")", at))
    depth = 0
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[at:j + 1]
    raise AssertionError("unbalanced braces")


def test_key_words_see_atomics_of_one_width():
    """The block trees lower a vertex's 64-bit word (key and pass mark) with
    atomicMin while other warps set and clear its prune bit: every atomic on
    the word has to be as wide, or they are not atomic to each other."""
    src = body("chl_build.cu", "team_kernel(TreeArgs a)")
    on_word = re.findall(r"atomic\w+\(\s*(?:kw|key_at|mark_at|\(uint32_t \*\))[^;]*;", src)
    assert len(on_word) >= 3
    for call in on_word:
        assert re.match(r"atomic\w+\(\s*kw \+ ", call), call


def test_line_order_is_not_read_from_a_lane_mask():
    """Lanes that __activemask() finds together in the line parser may be in
    different turns of its loop, so the lowest of them need not hold the
    smallest line: the first arc's line comes from every thread's own."""
    src = open(os.path.join(ROOT, "plant_gb300", "csrc", "chl_ingest.cu")).read()
    assert "__activemask()" in body("chl_ingest.cu", "take_slot(")
    assert "first_a" not in body("chl_ingest.cu", "take_slot(")
    assert src.count("atomicMin(&po->first_a") == 1
    parse = body("chl_ingest.cu", "parse_lines(")
    tail = parse[parse.rindex("kFailFormat"):]
    assert "__shfl_xor_sync(kFull, first_a" in tail and "atomicMin(&po->first_a, first_a)" in tail


def test_lazily_made_copies_are_published_whole():
    """Labels read from host memory are uploaded by their first query, and
    several queries may come first: one uploads, under a lock, and the pointer
    that the others test is set after the last copy.  (Shown by reading: a query
    that saw it earlier would walk memory that is not there yet.)"""
    up = body("chl_labels.cu", "labels_ensure_device(const chl_labels *L)")
    assert "lock_guard" in up and "&L->d_off" not in up and "&L->d_ent" not in up
    assert up.rindex("cudaMemcpy(") < up.rindex("L->d_ent =") < up.rindex("L->d_off =")
    down = body("chl_labels.cu", "labels_fetch_host(const chl_labels *l)")
    assert "lock_guard" in down and down.rindex("d2h_staged(") < down.rindex("l->host_valid = true")
    src = open(os.path.join(ROOT, "plant_gb300", "csrc", "chl_internal.h")).read()
    assert re.search(r"std::atomic<uint64_t \*> d_off", src) and re.search(r"std::atomic<bool> host_valid", src)
