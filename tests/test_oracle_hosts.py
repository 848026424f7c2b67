"""The recursive host programs (min-char-rnn, TreeLSTM) on the CPU oracle: sanity anchors that need no GPU.
An untrained classifier's loss is ln(classes) per prediction, and repeating one example must drive its loss down."""
import os

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ORA_HOSTS = os.path.join(ROOT, "oracle", "liblantern_oracle_hosts.so")


def _model(oracle_lib, name, batch):
    from lantern_b200.hosts import HostPrograms
    oracle_lib.set_math(0)
    return HostPrograms(oracle_lib, ORA_HOSTS, "orah_").model(name, batch, seed=42)


def test_rnn_untrained_loss_and_learning(oracle_lib):
    mark = oracle_lib.mark()
    T, V, B = 20, 80, 3
    m = _model(oracle_lib, "rnn", B)
    assert m.num_params == 5 and m.label_count == T * B and m.input_count == T * B * V
    ids = np.random.default_rng(0).integers(0, V, (T + 1, B))
    x = np.zeros((T, B, V), np.float32)
    x[np.arange(T)[:, None], np.arange(B)[None, :], ids[:T]] = 1.0
    y = ids[1:].astype(np.int32).ravel()
    first = m.step(x.ravel(), y, 0.01)
    assert abs(first - T * B * np.log(V)) < 0.02 * T * B * np.log(V)
    for _ in range(30):
        last = m.step(x.ravel(), y, 0.01)
    assert last < 0.5 * first
    m.close(); oracle_lib.reset(mark)


def test_treelstm_untrained_loss_and_learning(oracle_lib):
    from tests.test_gpu_models import _random_tree
    mark = oracle_lib.mark()
    m = _model(oracle_lib, "treelstm", 1)
    assert m.num_params == 22 and m.label_count == 1 + 4 * 99
    y = _random_tree(np.random.default_rng(4), 9)
    x = np.zeros(1, np.float32)
    first = m.step(x, y, 0.05)
    assert abs(first - 17 * np.log(5.0)) < 0.2
    for _ in range(8):
        last = m.step(x, y, 0.05)
    assert last < 0.1 * first
    m.close(); oracle_lib.reset(mark)


def test_treelstm_fused_gates_equal_operator_by_operator(oracle_lib):
    """One fused call per gate (affine_act) against the reference's operator-by-operator form on the oracle: same loss and
    the same 22 gradients up to the order of two float additions per gate."""
    from tests.test_gpu_models import _random_tree
    mark = oracle_lib.mark()
    y = _random_tree(np.random.default_rng(11), 7)
    x = np.zeros(1, np.float32)
    res = []
    for fused in (True, False):
        m = _model(oracle_lib, "treelstm", 1)
        m.use_fused_cells(fused)
        loss = m.step(x, y, 0.0, update=False)
        res.append((loss, [m.grad(i) for i in range(m.num_params)]))
        m.close(); oracle_lib.reset(mark)
    assert abs(res[0][0] - res[1][0]) <= 1e-6 * abs(res[1][0])
    for a, b in zip(res[0][1], res[1][1]):
        assert np.abs(a - b).max() <= 1e-5 * max(np.abs(b).max(), 1e-12)


@pytest.mark.parametrize("variant", ["treelstm", "treelstm_nips18"])
def test_treelstm_node_call_equals_operator_by_operator(oracle_lib, variant):
    """A whole tree node as one forward and one backward call (tree_node_fwd / tree_node_bwd) against the reference's
    operator-by-operator form, on the oracle, whose node entry points issue that operator sequence: same loss and the same 22
    gradients up to the order of a few float additions (both applications: exchanged roles with clipping, plain cell)."""
    from tests.test_gpu_models import _random_tree
    mark = oracle_lib.mark()
    x = np.zeros(1, np.float32)
    for leaves in (1, 2, 9, 30):
        y = _random_tree(np.random.default_rng(12 + leaves), leaves)
        res = []
        for level in (3, 2, 0):                      # the whole tree per call, a whole node per call, operator by operator
            m = _model(oracle_lib, variant, 1)
            m.use_fused_cells(level)
            loss = m.step(x, y, 0.0, update=False)
            res.append((loss, [m.grad(i) for i in range(m.num_params)]))
            m.close(); oracle_lib.reset(mark)
        for r in res[:2]:
            assert abs(r[0] - res[2][0]) <= 1e-6 * abs(res[2][0]), (leaves, r[0], res[2][0])
            for i, (a, b) in enumerate(zip(r[1], res[2][1])):
                assert np.abs(a - b).max() <= 1e-5 * max(np.abs(b).max(), 1e-12), (leaves, i)


def _labels(nodes, maxn=99):
    """Tree labels of the host program from (score, word, left, right) per node."""
    y = np.zeros(1 + 4 * maxn, dtype=np.int32)
    y[0] = len(nodes)
    for f in range(4):
        y[1 + f * maxn:1 + f * maxn + len(nodes)] = [node[f] for node in nodes]
    return y


GOOD_TREE = [(1, 0, 1, 2), (0, 7, -1, -1), (4, 0, 3, 4), (2, 999, -1, -1), (3, 5, -1, -1)]


@pytest.mark.parametrize("node,field,value", [(0, 0, 5), (3, 0, -1), (3, 1, 1000), (1, 1, -1), (2, 2, 5), (2, 3, 5), (2, 3, -1), (2, 2, 0), (2, 3, 2)])
def test_labels_that_are_no_tree_raise(oracle_lib, node, field, value):
    """A score outside the classes, a word outside the table, a child outside the tree and a circle: every way to issue a step raises, no
    parameter changes, and the program goes on working."""
    mark = oracle_lib.mark()
    m = _model(oracle_lib, "treelstm", 1)
    x, bad = np.zeros(1, np.float32), [list(v) for v in GOOD_TREE]
    bad[node][field] = value
    before = m.slab_params()
    for issue in (lambda: m.step(x, _labels(bad), 0.05), lambda: m.step_async(x, _labels(bad), 0.05), lambda: m.submit(x, _labels(bad), 0.05),
                  lambda: m.set_resident(x, _labels(bad))):
        with pytest.raises(RuntimeError, match="outside|descendant"):
            issue()
    assert np.array_equal(m.slab_params(), before)
    assert np.isfinite(m.step(x, _labels(GOOD_TREE), 0.05)) and not np.array_equal(m.slab_params(), before)
    m.close(); oracle_lib.reset(mark)


def test_submitted_trees_are_the_trees_of_their_steps(oracle_lib):
    """submit() puts the labels into a staging pair; the program builds the step from that pair, not from what a blocking step left behind."""
    from tests.test_gpu_models import _random_tree
    mark = oracle_lib.mark()
    rng, x = np.random.default_rng(8), np.zeros(1, np.float32)
    trees = [_random_tree(rng, leaves) for leaves in (3, 9, 2, 6)]
    runs = []
    for submit in (False, True):
        m = _model(oracle_lib, "treelstm", 1)
        m.step(x, trees[0], 0.05)
        runs.append([m.collect(m.submit(x, y, 0.05)) if submit else m.step(x, y, 0.05) for y in trees])
        m.close(); oracle_lib.reset(mark)
    assert runs[0] == runs[1]


# A part that node 0 does not reach and that is higher than its tree, a node 0 that is the child of another, a leaf and an inner node under
# two parents, one under the same parent twice.
ODD_TREES = [[(1, 0, 1, 2), (0, 7, -1, -1), (4, 3, -1, -1), (2, 0, 4, 5), (3, 5, -1, -1), (1, 0, 6, 7), (0, 9, -1, -1), (2, 11, -1, -1)],
             [(1, 8, -1, -1), (0, 0, 0, 2), (4, 3, -1, -1)],
             [(1, 0, 1, 2), (0, 0, 3, 4), (4, 0, 3, 5), (2, 6, -1, -1), (3, 5, -1, -1), (1, 2, -1, -1)],
             [(1, 0, 1, 2), (0, 0, 2, 3), (4, 0, 4, 5), (2, 6, -1, -1), (3, 5, -1, -1), (1, 2, -1, -1)],
             [(1, 0, 1, 1), (0, 0, 2, 3), (4, 1, -1, -1), (2, 6, -1, -1)]]


@pytest.mark.parametrize("variant", ["treelstm", "treelstm_nips18"])
@pytest.mark.parametrize("nodes", ODD_TREES, ids=["unreached", "child", "leaf shared", "node shared", "twins"])
def test_labels_that_are_more_or_less_than_a_tree(oracle_lib, variant, nodes):
    """The reference walks the arrays from node 0: a part it does not reach counts nothing, a node under two parents counts under both.
    The loss is that walk's (recomputed here from per-node losses of an untrained classifier) and every form of the program gives it."""
    mark = oracle_lib.mark()

    def count(i):
        return 1 + (0 if nodes[i][2] < 0 else count(nodes[i][2]) + count(nodes[i][3]))
    res = []
    for level in (3, 2, 1, 0):
        m = _model(oracle_lib, variant, 1)
        m.use_fused_cells(level)
        loss = m.step(np.zeros(1, np.float32), _labels(nodes), 0.0, update=False)
        res.append((loss, [m.grad(i) for i in range(m.num_params)]))
        m.close(); oracle_lib.reset(mark)
    assert abs(res[3][0] - count(0) * np.log(5.0)) < 0.01 * count(0)
    for r in res[:3]:
        assert abs(r[0] - res[3][0]) <= 1e-6 * abs(res[3][0])
        for i, (a, b) in enumerate(zip(r[1], res[3][1])):
            assert np.abs(a - b).max() <= 1e-5 * max(np.abs(b).max(), 1e-12), i


def test_rnn_fused_cell_equals_operator_by_operator(oracle_lib):
    """The recurrent cell and the output layer as one fused call each (affine_act_rows) against the operator-by-operator form."""
    mark = oracle_lib.mark()
    T, V, B = 20, 80, 3
    ids = np.random.default_rng(5).integers(0, V, (T + 1, B))
    x = np.zeros((T, B, V), np.float32)
    x[np.arange(T)[:, None], np.arange(B)[None, :], ids[:T]] = 1.0
    y = ids[1:].astype(np.int32).ravel()
    res = []
    for fused in (True, False):
        m = _model(oracle_lib, "rnn", B)
        m.use_fused_cells(fused)
        loss = m.step(x.ravel(), y, 0.0, update=False)
        res.append((loss, [m.grad(i) for i in range(m.num_params)]))
        m.close(); oracle_lib.reset(mark)
    assert abs(res[0][0] - res[1][0]) <= 1e-6 * abs(res[1][0])
    for a, b in zip(res[0][1], res[1][1]):
        assert np.abs(a - b).max() <= 2e-5 * max(np.abs(b).max(), 1e-12)


def test_rnn_whole_sequence_call_equals_operator_by_operator(oracle_lib):
    """The whole unrolled sequence as one forward and one backward call (rnn_seq_fwd / rnn_seq_bwd) against the
    operator-by-operator form, on the oracle, whose sequence entry points issue that very operator sequence: loss and the five
    gradients agree to the last bits of a few reordered float additions."""
    mark = oracle_lib.mark()
    T, V, B = 20, 80, 5
    ids = np.random.default_rng(6).integers(0, V, (T + 1, B))
    x = np.zeros((T, B, V), np.float32)
    x[np.arange(T)[:, None], np.arange(B)[None, :], ids[:T]] = 1.0
    y = ids[1:].astype(np.int32).ravel()
    res = []
    for level in (2, 0):
        m = _model(oracle_lib, "rnn", B)
        m.use_fused_cells(level)
        loss = m.step(x.ravel(), y, 0.0, update=False)
        res.append((loss, [m.grad(i) for i in range(m.num_params)]))
        m.close(); oracle_lib.reset(mark)
    assert abs(res[0][0] - res[1][0]) <= 1e-6 * abs(res[1][0])
    for a, b in zip(res[0][1], res[1][1]):
        assert np.abs(a - b).max() <= 2e-5 * max(np.abs(b).max(), 1e-12)


def test_deferred_zero_fill_is_invisible_on_the_oracle(oracle_lib):
    """The host programs declare large activation gradients unset (grad_unset) instead of taking them zero-filled; the CPU
    restatement keeps the reference's plain rule (it fills such a block with zeros at once), so a SqueezeNet step at batch 16
    (feature maps of 1.5 M floats and more) gives the same loss and the same gradients either way, bit for bit."""
    mark = oracle_lib.mark()
    rng = np.random.default_rng(3)
    x = rng.standard_normal(16 * 3072).astype(np.float32); y = rng.integers(0, 10, 16).astype(np.int32)
    res = []
    for deferred in (True, False):
        m = _model(oracle_lib, "squeezenet", 16)
        m.use_deferred_zero(deferred)
        loss = m.step(x, y, 0.0, update=False)
        res.append((loss, m.slab_grads()))
        m.use_deferred_zero(True)
        m.close(); oracle_lib.reset(mark)
    assert res[0][0] == res[1][0] and np.array_equal(res[0][1], res[1][1])


@pytest.mark.parametrize("batch", [1, 101, 252, 253, 505])
def test_submitted_batches_arrive_whole(oracle_lib, batch):
    """submit() copies a batch into its staging pair in pieces of 512 KB, those of 32 KB and more 64 bytes at a time: batches of one
    row (2,080 bytes), of 32 bytes more than a multiple of 64, of 128 bytes less than a piece, of a piece and 1,952 bytes and of two and 1,824 train as the blocking steps do, bit for bit, whatever the address of the array."""
    mark = oracle_lib.mark()
    rng = np.random.default_rng(batch)
    n = 20 * 26 * batch
    batches = [(rng.standard_normal(n + 1).astype(np.float32)[k % 2:n + k % 2], rng.integers(0, 26, 20 * batch).astype(np.int32)) for k in range(3)]
    res = []
    for feed in (False, True):
        m = _model(oracle_lib, "rnn_26_50", batch)
        if feed:
            losses = []
            for x, y in batches:
                losses.append(m.collect(m.submit(x, y, 0.01)))
        else:
            losses = [m.step(x, y, 0.01) for x, y in batches]
        res.append((losses, m.slab_params()))
        m.close(); oracle_lib.reset(mark)
    assert res[0][0] == res[1][0] and np.array_equal(res[0][1], res[1][1])


def test_programs_start_no_threads(oracle_lib):
    """Opening, stepping and closing a program costs no thread: neither the first step of a large batch nor the close of the last program
    may pay for helpers, and a process at its limit of threads must be able to train."""
    mark = oracle_lib.mark()
    rng = np.random.default_rng(1)
    x, y = rng.standard_normal(20 * 80 * 256).astype(np.float32), rng.integers(0, 80, 20 * 256).astype(np.int32)

    def threads():
        return len(os.listdir("/proc/self/task"))
    m = _model(oracle_lib, "rnn", 2)
    m.step(x[:20 * 80 * 2], y[:40], 0.01)                # the oracle's own OpenMP threads are there from now on
    m.close(); oracle_lib.reset(mark)
    before = threads()
    m = _model(oracle_lib, "rnn", 256)
    m.collect(m.submit(x, y, 0.01)); m.step(x, y, 0.01)
    assert threads() == before
    m.close(); oracle_lib.reset(mark)
    assert threads() == before
