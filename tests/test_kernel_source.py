"""Orders that kernels must keep and that no run can show (a store that comes
too early is lost only now and then): read from the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "belief-propagation_b200", "csrc")


def _code(name):
    """A source file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _body(code, start):
    """The brace-delimited body that follows the first match of `start`."""
    at = code.index("{", re.search(start, code).end())
    depth = 0
    for k in range(at, len(code)):
        depth += {"{": 1, "}": -1}.get(code[k], 0)
        if depth == 0:
            return code[at:k + 1]
    raise AssertionError("unbalanced braces")


def test_cluster_kernel_meets_before_it_touches_its_peers_shared_memory():
    """Distributed shared memory is defined only once every block of the
    cluster has started, which a cluster barrier shows."""
    body = _body(_code("batch_cluster.cuh"), r"k_batch_cluster\(")
    assert "map_shared_rank" in body
    assert "cluster.sync()" in body[:body.index("map_shared_rank")]


def test_serial_launches_take_their_own_residency():
    """A persistent grid larger than the kernel's own resident blocks runs as a
    full wave and a partial one: the serial-delta form's grid is asked of the
    serial-delta form."""
    body = _body(_code("loopy.cu"), r"static int block_tiles\(")
    serial = body[body.index("else if (serial)"):]
    assert re.search(r"resident_blocks_mb<MS, UNI, FU, flood_min_blocks_serial<MS, FU>\(\), true>", serial)


def test_split_passes_of_small_graphs_do_not_overlap():
    """Two kernels of less than a wave each then wait for each other's blocks: a
    quarter of an iteration of 50,000 nodes."""
    body = _body(_code("loopy.cu"), r"static int split_run_nv\(")
    assert re.search(r"overlap = grid_for\(g->V, kNodeThreads\) >= 4u \* gb", body)
    assert len(re.findall(r"Threads, overlap, g->stream", body)) == 2


def test_forward_without_stored_messages_keeps_large_blocks():
    """From 5 states on 128 threads cost it a twelfth of its time."""
    code = _code("unrolled.cu")
    assert re.search(r"stored \|\| S <= 4 \? u_threads\(V\) : \(unsigned\)kUThreads", code)
    assert "u_fwd_threads<S>(u->V, u->ms.n != 0)" in _body(code, r"static int u_forward\(")


def test_network_blocks_of_ten_states_divide_in_fp32():
    """The f64 quotients cost a twentieth of a batch's time there."""
    code = _code("batch.cu")
    assert "S == 10" in _body(code, r"constexpr bool block_divides_f32\(")
    assert code.count("send_msg<S, true, block_divides_f32<S>()>(") == 2


def test_two_table_adjoint_multiplies_in_fp32():
    """Its scatter form multiplies fp32 operands; split into two TF32 parts
    without their low product they carry up to seven times the error."""
    body = _body(_code("unrolled.cu"), r"k_u_bwd_pull2\(")
    assert "tf32" not in body and "mma" not in body.lower()
