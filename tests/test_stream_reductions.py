"""CPU check of the order in which the single-session decode kernel's warps share `DsShared::red`: an array that is read after a barrier may
be written again only behind another barrier.  The kernel's source is walked along the paths a unit can take, twice in a row, as a list
of barriers, writes and reads."""
import os
import re

from conftest import ROOT

EVENT = re.compile(r"ds_block_sum\([^;]*?S->red\[(?P<sum>\d)\]|S->red\[(?P<write>\d)\]\[w\]\s*=(?!=)|S->red\[(?P<read>\d)\]|ds_consumer_sync(?:_or)?\(|bar_arrive\(\)|bar_wait\(\)")


def _events(text):
    out = []
    for m in EVENT.finditer(re.sub(r"//[^\n]*", "", text)):
        if m["sum"]:  # write, barrier, read
            out += [("write", m["sum"]), ("barrier", ""), ("read", m["sum"])]
        elif m["write"]:
            out.append(("write", m["write"]))
        elif m["read"]:
            out.append(("read", m["read"]))
        else:
            out.append(("barrier", ""))
    return out


def _unsafe(events):
    pending, bad = set(), []  # arrays read since the last barrier
    for kind, a in events:
        if kind == "barrier":
            pending.clear()
        elif kind == "read":
            pending.add(a)
        elif a in pending:
            bad.append(a)
    return bad


def _sections():
    src = open(os.path.join(ROOT, "rwkv-rsv_b200", "csrc", "decode_stream.cuh")).read()
    body = src[src.index("for (int u = 0; u < 4 * L"):src.index("every CTA reduces the candidates itself")]
    cut = ["if (ln) {", "} else if (ph == 1) {", "---- operands: one scale per vector", "---- rows, in batches of tiles", "phase 2: one CTA per head", "the token's one grid barrier",
           "} else {\n                // arg-max"]
    at = [body.index(c) for c in cut]
    assert at == sorted(at)
    ln, other, operands, rows, heads, plain, argmax = [_events(body[a:b]) for a, b in zip(at, at[1:] + [len(body)])]
    assert any(k == "barrier" for k, _ in rows) and any(k == "write" for k, _ in heads)
    rows = [("barrier", "")]  # (between batches; a unit has one at least, after its products)
    return ln, other, operands, rows, heads, plain, argmax


def test_no_array_is_written_while_another_warp_may_read_it():
    ln, other, operands, rows, heads, plain, argmax = _sections()
    unit_ln, unit = ln + operands + rows, other + operands + rows
    head_rows = ln + operands  # a CTA without rows of the vocabulary head
    layer = [unit_ln + h + unit + unit_ln + unit for h in ([], heads)]
    for a in layer:
        for b in layer:
            for end in (unit_ln + plain, head_rows + plain, unit_ln + argmax, head_rows + argmax):
                # (a token begins with a barrier)
                assert not _unsafe(a + b + end + [("barrier", "")] + a + b), "written again without a barrier in between"


def test_the_walk_sees_a_missing_barrier():
    # the order the kernel had once: a head's last sum and the second operand maximum in the same array
    ln, other, operands, rows, heads, *_ = _sections()
    shared = [(k, "3" if a == "5" else a) for k, a in operands]
    assert _unsafe(ln + shared + rows + heads + other + shared) == ["3"]
