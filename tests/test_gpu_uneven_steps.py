"""Steps whose requests differ much in length, through the runner: the decode attention gives long contexts more key
slices there, in graphs of their own where that is another kernel.  Decode and mixed steps with and without graphs, step
after step as lengths change and as the batch flips between uneven and even, against the plain implementation; and
that buffers stay where they are and no graph is captured that is not needed."""
import numpy as np
import pytest
import torch

import plain_hunyuan as ph
import tiny_configs
import trace_tools as tt

pytestmark = pytest.mark.gpu

# 8 key/value heads of 128: from 9 requests on (a bucket of 16) two key slices each, more for long contexts among short ones
CFG = dict(tiny_configs.A, vocab_size=301, hidden_size=256, intermediate_size=384, num_attention_heads=16,
           num_key_value_heads=8, head_dim=128, max_position_embeddings=2048)
SHORT, LONG = [20, 33, 60, 5, 47, 28, 31, 52, 16, 40], [900, 700, 600]


class Run:
    """A runner, and for every request its tokens and the plain logits of all its places."""

    def __init__(self, monkeypatch, folder, seqs=(), plain=(), **opts):
        from crane_b200.generation import ModelForCausalLM
        opts = dict(dict(page_size=64, num_pages=200, max_concurrent=32, max_batched_tokens=1024, chunk_size=1024), **opts)
        self.model = ModelForCausalLM.from_pretrained(folder, "bf16", **opts)
        self.r, self.seqs, self.plain = self.model.runner, seqs, plain
        self.at = {i: 0 for i in range(len(seqs))}
        self.balanced = {"fused": 0, "plain": 0}
        k = self.r.rt.kernels
        for kind, name in (("fused", "paged_decode_attention_fused"), ("plain", "paged_decode_attention")):
            monkeypatch.setattr(k, name, self._counted(getattr(k, name), kind))

    def _counted(self, inner, kind):
        def call(*a, **kw):
            self.balanced[kind] += kw.get("balance") is not None
            return inner(*a, **kw)
        return call

    def step(self, counts, check=True):
        """counts: {request: tokens of it}; the logits of every request's last place."""
        from crane_b200.engine import StepEntry
        entries = []
        for i, n in counts.items():
            entries.append(StepEntry(i, self.seqs[i][self.at[i]:self.at[i] + n], [n - 1]))
            self.at[i] += n
        got = self.r.step(entries)
        if check:
            self.compare(got, [(i, self.at[i] - 1) for i in counts])
        return got

    def compare(self, got, places):
        want = np.stack([self.plain[i][p] for i, p in places])
        got = got.float().cpu().numpy()
        assert got.shape == want.shape and np.isfinite(got).all()
        worst = np.abs(got - want).max(axis=1) / np.abs(want).max()
        assert worst.max() < tt.TOL["bfloat16"], (places[int(worst.argmax())], worst.max())

    def prefill(self, who, lens):
        small = {i: n for i, n in zip(who, lens) if n < 100}
        for i, n in zip(who, lens):
            if n >= 100:
                self.step({i: n})
        if small:
            self.step(small)

    def done(self):
        self.r.rt.check_errors()
        for i, n in self.at.items():
            if n:
                self.r.end(i)
        self.r.table.check()


@pytest.fixture(scope="module")
def uneven_model(tmp_path_factory):
    from crane_b200.weights.random_init import write_model_folder
    folder = write_model_folder(str(tmp_path_factory.mktemp("uneven")), CFG, 3, "bfloat16", std=0.05, norm_std=0.05)
    return make(folder, 24)


def make(folder, n):
    cfg, w = ph.load_folder(folder)
    rng = np.random.default_rng(5)
    seqs = [rng.integers(0, cfg.vocab_size, 1000 if i >= len(SHORT) - 2 else 120).tolist() for i in range(n)]
    plain = [ph.logits_all(cfg, w, s) for s in seqs]
    return folder, seqs, plain


@pytest.mark.parametrize("graphs", [False, True])
def test_uneven_steps_match_the_plain_logits(uneven_model, monkeypatch, graphs):
    run = Run(monkeypatch, *uneven_model, use_cuda_graphs=graphs)
    short, long_ = list(range(10)), [10, 11, 12]
    run.prefill(short + long_, SHORT + LONG)
    every = {i: 1 for i in short + long_}
    for _ in range(3):
        run.step(every)                                     # 13 requests, uneven
    assert run.balanced["fused"] > 0
    for _ in range(3):
        run.step({i: 1 for i in short})                     # 10 requests of the same bucket, even
    for _ in range(2):
        run.step(every)
    run.step({9: 600})                                      # a short one grows: the lengths change under the graph
    for _ in range(2):
        run.step(every)
    for t in range(4):                                      # beside a prompt, which ends with the step
        run.step({**every, 13 + t: 30 + t})
        run.r.end(13 + t)
        run.at[13 + t] = 0
    assert run.balanced["plain"] > 0
    for _ in range(2):
        run.step({i: 1 for i in [8, 9] + long_ + short[:6]})     # another composition of the bucket
    assert (run.r.graph_replays > 0) == graphs
    run.done()


def test_buffers_stay_where_they_are(model_folders, monkeypatch):
    """Steps of changing size at model layer sizes: a buffer that grows would throw all graphs away."""
    from crane_b200.engine import StepEntry
    run = Run(monkeypatch, model_folders("S18", "bfloat16"), max_concurrent=20)
    r, rng = run.r, np.random.default_rng(1)
    draw = lambda n: rng.integers(0, 1000, n).tolist()      # noqa: E731
    for i, n in enumerate((250, 137, 192, 193, 40, 300, 700) + (30,) * 9):
        r.step([StepEntry(i, draw(n), [n - 1])])
    assert r.rt.ws.generation == 0
    r.step([StepEntry(0, draw(1), [0])])
    kept = len(r._graphs)
    assert kept >= 1
    singles = [StepEntry(i, draw(1), [0]) for i in range(16)]
    r.step(singles)                                         # 16 requests of very different lengths
    for _ in range(2):
        r.step([StepEntry(i, draw(1), [0]) for i in range(16)] + [StepEntry(16, draw(200), [199])])
        r.end(16)
    assert run.balanced["plain"] > 0
    assert r.rt.ws.generation == 0 and len(r._graphs) > kept
    run.done()
    for i in range(16):
        r.end(i)


def decode_graphs(r):
    return [k for k in r._graphs if isinstance(k, int)]


@pytest.mark.parametrize("change,n", [(dict(num_key_value_heads=4), 3), (dict(head_dim=64), 9)])
def test_no_second_graph_of_the_same_kernels(change, n, tmp_path, monkeypatch):
    """Three requests at four key/value heads take 8 key slices each however long they are, and at head size 64 nothing is
    balanced: steps of even and of uneven lengths replay one graph."""
    from crane_b200.engine import StepEntry
    from crane_b200.weights.random_init import write_model_folder
    folder = write_model_folder(str(tmp_path / "m"), dict(CFG, **change), 3, "bfloat16", std=0.05, norm_std=0.05)
    run = Run(monkeypatch, folder)
    r = run.r
    for i in range(2 * n):
        r.step([StepEntry(i, [(7 * j + i) % 300 for j in range(700 if i == 0 else 20 + i)], [])])
    before = r.graph_replays
    for _ in range(3):
        for first in (0, n):                                # n requests with the long one, then n without
            r.step([StepEntry(i, [5], [0]) for i in range(first, first + n)])
    assert run.balanced == {"fused": 0, "plain": 0}
    assert len(decode_graphs(r)) == 1 and r.graph_replays == before + 5
    run.done()
    for i in range(2 * n):
        r.end(i)


def test_balanced_and_windowed_attention_in_one_step(monkeypatch):
    """Layers that alternate between all earlier positions and a window of 100: lengths of 5 to 900 are balanced in the former
    and equal enough in the latter; decode and mixed steps against the plain computation."""
    import test_gpu_window_layers as tw
    from crane_b200.config import EngineConfig, resolve
    from crane_b200.engine import ModelRunner, StepEntry
    from crane_b200.parts import model_manifest
    from crane_b200.weights.random_init import random_tensors
    cfg = dict(tw.CFG, hidden=128, heads=16, kv_heads=8, head_dim=128, window=100, max_pos=1024, layers=2)
    monkeypatch.setattr(tw, "CFG", cfg)
    tw.register()
    tensors = random_tensors(model_manifest(resolve(cfg).build_spec(cfg)), 9, torch.bfloat16, std=0.08, norm_std=0.05)
    w = {k: v.double().numpy() for k, v in tensors.items()}
    r = ModelRunner(None, EngineConfig(dtype="bfloat16", page_size=32, num_pages=200, max_concurrent=20,
                                       max_batched_tokens=1024), config=cfg, tensors=tensors)
    rng = np.random.default_rng(2)
    lens = SHORT + LONG
    seqs = [rng.integers(0, 120, n + 10).tolist() for n in lens]
    want = [tw.plain_logits(w, s) for s in seqs]
    forms = []
    prepare = r.prepare
    monkeypatch.setattr(r, "prepare", lambda *a, **kw: forms.append(prepare(*a, **kw)) or forms[-1])

    def check(got, places):
        for g, (i, p) in zip(got.float().cpu().numpy(), places):
            assert np.abs(g - want[i][p]).max() / np.abs(want[i]).max() < 3e-2, (i, p)
    for i, n in enumerate(lens):
        check(r.step([StepEntry(i, seqs[i][:n], [n - 1])]), [(i, n - 1)])
    for t in range(6):
        entries = [StepEntry(i, [seqs[i][n + t]], [0]) for i, n in enumerate(lens)]
        if t >= 3:
            entries.append(StepEntry(50 + t, seqs[10][:40], []))
        check(r.step(entries), [(i, n + t) for i, n in enumerate(lens)])
        assert {k[3]: f for k, f in forms[-1].decode_forms.items()} == {0: 1, 100: 0}
    r.rt.check_errors()
    for i in list(range(len(lens))) + [53, 54, 55]:
        r.end(i)
    r.table.check()


def test_a_batch_that_crosses_the_line_keeps_its_graph_at_first(uneven_model, monkeypatch):
    """Steps of ten requests that turn uneven replay the graph their bucket has; the balanced one is captured when they have
    come often.  The same the other way round, in a bucket that has the balanced graph alone."""
    run = Run(monkeypatch, *uneven_model)
    r, short, long_ = run.r, list(range(10)), [10, 11, 12]
    run.prefill(short + long_, SHORT + LONG)
    even, uneven = {i: 1 for i in short[:9]}, {i: 1 for i in short[:6] + long_}
    captures = r.graph_captures
    run.step(even)
    assert r.graph_captures == captures + 1
    for t in range(1, r.CAPTURE_BUSY):
        run.step(uneven)
        assert r.graph_captures == captures + 1 and run.balanced["fused"] == 0
    run.step(uneven)
    assert r.graph_captures == captures + 2 and run.balanced["fused"] > 0
    replays = r.graph_replays
    for _ in range(3):
        run.step(uneven)
        run.step(even)
    assert (r.graph_captures, r.graph_replays) == (captures + 2, replays + 6) and len(decode_graphs(r)) == 2
    for k in decode_graphs(r):                              # (as in an engine that has met uneven steps only)
        if k < 1 << 21:
            del r._graphs[k]
    for _ in range(3):
        run.step(even)
    assert r.graph_captures == captures + 2
    run.done()


def test_replay_while_the_device_is_busy(uneven_model, monkeypatch):
    """Short prompts one after the other without a look at their results: a shape is captured on a busy device when it has
    come 16 times, not before, and then replayed; up to 16 tokens are padded to 16 rows.  The logits are the plain ones."""
    class Busy:
        def query(self):
            return False

        def record(self):
            pass
    run = Run(monkeypatch, *uneven_model)
    r = run.r
    monkeypatch.setattr(r, "_step_done", Busy())
    kept = []
    for t in range(30):
        i, n = t % len(run.seqs), 1 + (7 * t) % 16
        if n == 1:
            n = 16                                          # (single tokens are decode steps)
        kept.append((run.step({i: n}, check=False).clone(), [(i, n - 1)]))
        r.end(i)
        run.at[i] = 0
        assert r.graph_captures == (1 if t >= 15 else 0)
    assert r.graph_replays == 14 and [k[:2] for k in r._graphs] == [("rows", 16)]
    for got, places in kept:
        run.compare(got, places)
    run.done()
