"""What device code has to keep to on its failure paths, held against its source: a wait of a kernel on its own copies cannot be
made to run out on a GPU that works (a look at a barrier suspends the thread for longer than a copy takes: with a limit of one
clock none of 300 launches gave up)."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "orca_b200", "csrc")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("name,done", [("attn_query.cu", "accfull"), ("attn_out.cu", "acc2"), ("gru_rows.cu", "accfull"),
                                       ("score_rows.cu", "accfull")])
def test_a_warp_that_gives_up_stops_and_waits_for_what_it_has_in_flight(name, done):
    """A copy thread whose slot is not handed back issues no further copy into it (nor arrives twice on its barrier), the
    products stop likewise, and copies and products are waited for before shared and tensor memory are given up."""
    text = _source(name)
    copies, rest = text.split("if (warp == 0) {", 1)[1].split("} else if (warp == 1) {", 1)
    products = rest.split("} else {", 1)[0]
    at = [copies.index(x) for x in ("; alive && ", "mbar_wait(empty(", "if (!alive) break;", "mbar_expect_tx(full(", "mbar_settle(full(")]
    assert at == sorted(at)
    assert "if (alive) mma_commit(empty(s));" in products and re.search(r"[^(] mma_commit\(empty", products.replace("if (alive) ", "(")) is None
    assert products.rindex(f"mma_commit({done})") < products.index(f"mbar_settle({done}, (t - 1) & 1)")


def test_a_query_that_did_not_come_is_waited_for():
    text = _source("attention.cu")
    at = [text.index(x) for x in ("mbar_wait(qbar, phase", "phase ^= alive;", "if (!alive) tc::mbar_settle(qbar, phase);")]
    assert at == sorted(at)


def test_no_entry_point_drops_the_status_word_it_is_given():
    """Every entry point that takes one hands it to what it launches: its kernels have nothing else to say that rows are wrong."""
    for name in os.listdir(CSRC):
        assert name.endswith((".cu", ".cuh")) is False or "(void)d_status" not in _source(name), name
