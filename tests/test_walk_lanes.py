"""The walk's lanes share the walk's stacks: what lane 0 stores, all read.  Between a read and
the next store to the same place, and the other way round, the whole warp has to meet, or a
lane that falls behind goes on with another frame.  The kernel's own text runs here on the
host with one coroutine per lane (tests/cpp/walk_lanes.cpp), lane 0 ahead of all others and
behind them: the same pieces and contigs must come out."""
import os
import re
import subprocess

import pakman_plus_gb300

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = os.path.join(os.path.dirname(pakman_plus_gb300.__file__), "csrc", "pk_compact.cu")


def _definition(text, head):
    """The definition whose first line holds `head`, its template line before it included."""
    at = text.index(head)
    start = text.rindex("\n", 0, at) + 1
    before = text[:start].rstrip("\n").rsplit("\n", 1)[-1]
    if before.startswith("template"):
        start -= len(before) + 1
    depth, i = 0, text.index("{", at)
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            break
    return text[start:i] + (";" if text[i] == ";" else "") + "\n"


def _extract():
    text = open(SOURCE).read()
    out = ["typedef unsigned __int128 u128;\n"]
    for name in ("kTerm", "kLenMask", "kWalkMaxBases", "kNoNode"):
        out.append(re.search(r"^constexpr \w+ %s = .*$" % name, text, re.M).group(0) + "\n")
    out.append(_definition(text, "enum : uint32_t {"))
    for name in ("Side", "WStep", "WResume", "WPath", "WPiece", "WContig"):
        out.append(_definition(text, "struct %s {" % name))
    for head in ("KeyT low_mask(", "uint64_t key_bases(", "WStep ld_step(", " k_walk("):
        out.append(_definition(text, head))
    return "".join(out)


def test_walk_is_the_same_for_any_order_of_lanes(tmp_path):
    (tmp_path / "walk_extract.h").write_text(_extract())
    exe = str(tmp_path / "walk_lanes")
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", str(tmp_path), "-o", exe,
                    os.path.join(HERE, "cpp", "walk_lanes.cpp")], check=True, capture_output=True, text=True)
    first, last = (subprocess.run([exe, order], check=True, capture_output=True, text=True).stdout
                   for order in ("first", "last"))
    assert last.startswith("recorded err 0 contigs 6 ")
    assert first == last
