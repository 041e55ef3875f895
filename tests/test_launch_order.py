"""Kernels that are launched as programmatic dependents wait for their predecessor on every way out: a kernel that leaves without waiting may
complete before it, and the launch behind, which waits for this kernel alone, then runs beside the one in front.  Read from the sources: such an
overlap of two kernels on one buffer cannot be provoked safely."""
import glob
import os
import re

import pytest

import __graft_entry__ as entry

CSRC = os.path.join(entry.PKG_DIR, "csrc")


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced source")


def _sources():
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        out[os.path.basename(path)] = re.sub(r'"(\\.|[^"\\\n])*"', '""', text)
    return out


SOURCES = _sources()


def _without_lambdas(text):
    for m in reversed(list(re.finditer(r"\[&?\]\s*\([^()]*\)\s*(->\s*\w+\s*)?(?=\{)", text))):
        text = text[:m.end()] + text[_closing(text, m.end(), "{}") + 1:]
    return text


def _kernels(text):
    """name -> body of every kernel of a file, its lambdas left out"""
    found = {}
    for m in re.finditer(r"__global__", text):
        head = re.compile(r"\b(?!__launch_bounds__)(\w+)\s*\(").search(text, re.compile(r"(__launch_bounds__\s*\([^()]*(\([^()]*\)[^()]*)*\))?").match(
            text, re.compile(r"__global__\s*(void)?\s*").match(text, m.start()).end()).end())
        args = _closing(text, head.end() - 1, "()")
        opens = text.find("{", args)
        if text[args + 1:opens].strip() == "":
            found[head.group(1)] = _without_lambdas(text[opens:_closing(text, opens, "{}") + 1])
    return found


KERNELS = {(f, n): body for f, text in SOURCES.items() for n, body in _kernels(text).items()}
WAIT = re.compile(r"\b(pdl_wait|pdl_enter|rows_enter)\s*\(")


def _dependents():
    """Kernels that a file names in a launch as programmatic dependent."""
    out = []
    for f, text in SOURCES.items():
        for m in re.finditer(r"\blaunch_pdl\w*\s*\(", text):
            call = text[m.start():_closing(text, m.end() - 1, "()")]
            out += [(f, n) for ff, n in KERNELS if ff == f and re.search(rf"\b{n}\b", call)]
    return sorted(set(out))


def test_the_sources_are_read():
    assert len(KERNELS) > 60 and len(_dependents()) > 25
    assert {("la_kernels.cu", "la_decode_kernel"), ("gemm_rows.cu", "rows_stream_kernel"), ("fa_decode.cu", "fa_decode_split_kernel")} <= set(_dependents())


@pytest.mark.parametrize("file,name", sorted(set(_dependents()) | {k for k, b in KERNELS.items() if WAIT.search(b)}))
def test_no_way_out_before_the_wait(file, name):
    body = KERNELS[file, name]
    wait = WAIT.search(body)
    assert wait, "launched as a programmatic dependent, never waits"
    assert not re.search(r"\breturn\s*;", body[:wait.start()]), "leaves before it waits for its predecessor"


@pytest.mark.parametrize("file,name", sorted(k for k, b in KERNELS.items() if "pdl_launch_dependents" in b or "rows_enter" in b))
def test_the_next_launch_is_let_in_behind_the_wait(file, name):
    """... or through rows_enter, which keeps that order for launches that ask for it."""
    body = KERNELS[file, name]
    lets = body.find("pdl_launch_dependents")
    assert lets < 0 or WAIT.search(body).start() < lets


@pytest.mark.parametrize("file,name", [("gemm_rows.cu", "rows_wide_kernel"), ("gemm_rows.cu", "rows_stream_kernel"), ("gemm_rows.cu", "rows_deep_kernel"),
                                       ("la_chunk.cu", "la_chunk_own_kernel"), ("la_chunk.cu", "la_chunk_walk_kernel")])
def test_a_wait_that_runs_out_leaves_no_copy_behind(file, name):
    """A CTA that gives up waits once more for its copies: its shared memory may be another's as soon as it leaves."""
    assert "mbar_drain" in KERNELS[file, name]
