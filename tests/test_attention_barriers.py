"""Order of the barriers of the dK / dV kernel, read from its source: what no run shows, because only an unlucky delay of a
warp or of the issuing thread would break it."""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "nabla_b200" / "csrc" / "attention_tcgen05.cu"


def _kernel():
    text = SOURCE.read_text()
    body = text[text.index("attn_bwd_dkdv_kernel(const __grid_constant__"):]
    body = body[: body.index("\n}\n")]
    issuer = body[body.index("} else if (warp == 1) {"): body.index("} else if (warp >= 4) {")]
    issuer = issuer[issuer.index("for (int it = 0; it < n_it"):]
    threads = body[body.index("} else if (warp >= 4) {"):]
    return issuer, threads[threads.index("for (int it = 0; it < n_it"): threads.index("if (ok && n_it > 0)")]


def _issuer_order(regions):
    """{"wait x" / "commit x": place in the issuing thread's loop body} of the form with that many score regions."""
    at = {}
    for m in re.finditer(r"(?:NREG == (\d) (&&|\|\|) !?)?(mbar_wait|umma_commit)\(&?(\w+)", _kernel()[0]):
        form, op, call, name = m.groups()
        if form is not None and (int(form) == regions) != (op == "&&"):
            continue
        at[("wait " if call == "mbar_wait" else "commit ") + name] = m.start()
    return at


@pytest.mark.parametrize("regions", [2, 3])
@pytest.mark.parametrize("release,read", [("do_empty", "nd2["), ("q_empty", "nl2[")])
def test_statistics_of_a_stage_are_read_before_it_is_loaded_again(regions, release, read):
    """A stage may be given back only behind a barrier on which the threads arrive after their last read of it."""
    order, threads = _issuer_order(regions), _kernel()[1]
    later = [b for b in ("p_full", "ds_full") if threads.index(f"mbar_arrive({b})") > threads.rindex(read)]
    assert later and any(order[f"wait {b}"] < order[f"commit {release}"] for b in later)


@pytest.mark.parametrize("regions", [2, 3])
@pytest.mark.parametrize("barrier,published", [("p_full", "s_full"), ("ds_full", "dp_full"), ("dp_read", "dp_full")])
def test_issuer_looks_at_a_barrier_before_the_threads_can_arrive_for_the_next_tile(regions, barrier, published):
    """Threads arrive for the next tile once ``published`` of it is there; a second arrival of all flips the parity that the
    issuer's wait for this tile looks for."""
    order, threads = _issuer_order(regions), _kernel()[1]
    assert threads.index(f"mbar_wait({published}") < threads.index(f"mbar_arrive({barrier})")
    if barrier == "dp_read" and regions == 3:
        assert "wait dp_read" not in order
    else:
        assert order[f"wait {barrier}"] < order[f"commit {published}"]
