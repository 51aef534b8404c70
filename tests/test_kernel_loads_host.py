"""Loads through the read-only path (__ldg and its variants) ask for memory that
nobody writes while the kernel runs.  The iterations' kernels may start while the
one before still runs, so only what is constant over those kernels may be read
so: the tets' records, the index tables, the materials, a finished tape.  This
reads the kernels' sources and looks at every such load's operand."""
import glob
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rdc-xpbd-taichi_gb300", "csrc")

CONSTANT = {
    # records and materials
    "tets", "dm_a", "dm_b", "dm_c", "v0", "lid", "tinv_mu", "tinv_la", "inv_mu", "inv_la",
    # index tables
    "v2t_off", "v2t_slot", "voff", "pverts", "pv_start", "patch_body", "patch_ntets", "vblock_body", "body_tets",
    "body_patches", "body_vblocks", "body_first", "body_vfirst", "corners", "cs", "pv", "ex", "dst", "dst_off", "inbox",
}
# local names: a slice of pv_slots, and the tape rows that the reverse kernels read
LOCAL = {"src": "d.pv_slots", "X": "tp."}


def _calls(text):
    """(function, argument text) of every read-only load."""
    for m in re.finditer(r"\b(__ldg|ldg_hint|ldg_pair)\(", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), text[m.end():k - 1]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(SRC, "*.cu*"))), ids=os.path.basename)
def test_read_only_loads_are_of_constant_memory(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    # the loads' own definitions
    text = re.sub(r"__device__ __forceinline__ \w+ (?:ldg_hint|ldg_pair)\([^)]*\)", "", text)
    for name, arg in _calls(text):
        a = re.sub(r"reinterpret_cast<[^>]*>", "", arg)
        member = re.search(r"\b(?:\w+\.)*(?:\w+->)*(\w+)", a.replace("&", " ").strip(" (")).group(1)
        if name == "__ldg" and arg in ("p", "p + 1"):  # the body of a helper
            continue
        if member in LOCAL:
            uses = re.findall(r"\* %s = ([^;]*);" % member, text)
            assert uses and all(LOCAL[member] in u for u in uses), (name, arg, uses)
        else:
            assert member in CONSTANT, (name, arg)


def test_lists_and_positions_have_ordinary_loads():
    text = open(os.path.join(SRC, "xpbd_batch.cu")).read()
    for read in ("&d.ctl->n_act_patches[d.stop_par]", "d.act_patch[d.stop_par] + p", "&d.ctl->n_act_patches[a.par]",
                 "list + c0", "&d.ctl->n_act_vblocks[u.par]", "P + g"):
        assert "ld_prev(%s)" % read in text, read
    text = open(os.path.join(SRC, "xpbd_device.cuh")).read()
    for body in re.findall(r"ld_prev\(const \w+\* p\) \{(.*?)\n\}", text, re.S):
        assert "asm volatile(\"ld.global." in body and ".nc" not in body  # stays behind the wait, itself volatile
