"""What the native library decides on the host, called without a GPU."""
import ctypes
import threading

import pytest

from openinfer_b200.kernels import lib as klib
from openinfer_b200.kernels import native


def _averages_behind(terms, layer, results):
    """Indexes of the layers whose averages layer ``layer`` adds up terms for; ``terms``: what each layer averages (None: nothing)."""
    layers = (native.BranchLayerDesc * len(terms))()
    for i, t in enumerate(terms):
        if t is not None:
            layers[i].depth_coef, layers[i].depth_terms, layers[i].depth_dtype = 1000 + i, t, i % 2
    d = native.DepthAhead()
    assert klib.load().oi_depth_ahead_layers(layers, len(terms), layer, results, ctypes.byref(d)) == 0
    chosen = [d.coef[q] - 1000 for q in range(d.next)]
    assert [d.coef_dtype[q] for q in range(d.next)] == [i % 2 for i in chosen]
    return chosen


@pytest.mark.parametrize("terms,layer,results,want", [
    (list(range(2, 12)), 3, 4, [4, 5, 6]),
    (list(range(2, 12)), 7, 8, [8, 9]),                                # fewer than three layers left
    (list(range(2, 12)), 9, 10, []),
    ([2, 3, None, 4, 5, None, 6, None, 7, 8], 4, 4, [6, 8, 9]),        # layers in between that average nothing
    ([2, 3, 4, 5, 6, 3, 8, 9, 10, 11], 3, 4, [4]),                     # coefficients fewer than their turn asks for: not read
    ([2, 3, 4, 5, 5, 7, 8, 9, 10, 11], 3, 4, []),
])
def test_sums_ahead_are_of_averages_whose_coefficients_are_all_there(terms, layer, results, want):
    assert _averages_behind(terms, layer, results) == want


def test_slots_are_cleared_on_the_tensors_own_device(monkeypatch):
    """The calling thread's current device may be another than the cache's."""
    import torch

    from openinfer_b200.kernels import ops
    current, launched = ["another device"], []

    class Device:
        def __init__(self, device):
            self.device = device

        def __enter__(self):
            self.was, current[0] = current[0], self.device

        def __exit__(self, *exc):
            current[0] = self.was

    class Library:
        @staticmethod
        def oi_clear_slots(table, tensors, max_bytes, slot, stream):
            launched.append((current[0], stream, slot, tensors, max_bytes))
            return 0

    monkeypatch.setattr(torch.cuda, "device", Device)
    monkeypatch.setattr(ops, "_cuda", lambda *tensors: None)
    monkeypatch.setattr(ops, "_stream", lambda: f"stream of {current[0]}")
    monkeypatch.setattr(ops._lib, "current_device", lambda: 1)
    monkeypatch.setattr(ops._lib, "load", lambda: Library)
    ops.SlotClearer([torch.ones(4, 3), torch.ones(4, 2, 8)]).clear(2)
    assert launched == [(torch.device("cpu"), "stream of cpu", 2, 2, 64)]
    assert current[0] == "another device"


def test_a_launch_fence_belongs_to_the_thread_that_asked_for_it():
    """Between a step's metadata and its first kernel another thread may launch (it opens a request): that launch does not use up the
    plain order which the step's first kernel was to get."""
    L = klib.load()
    seen = []

    def other():
        seen.append(L.oi_launch_fence_pending())

    def asks():
        L.oi_launch_fence()
        t = threading.Thread(target=other)
        t.start()
        t.join()
        seen.append(L.oi_launch_fence_pending())

    t = threading.Thread(target=asks)       # a thread of its own: this test's fence reaches no launch
    t.start()
    t.join()
    assert seen == [0, 1]


@pytest.mark.parametrize("stream,few,want", [(0, 0, 0), (2, 0, 2), (0, 1, 101), (3, 2, 3)])
def test_the_decode_products_status_is_both_kernels(monkeypatch, stream, few, want):
    """Which of the two kernels took a product is the dispatch's affair: one question covers both."""
    from openinfer_b200.kernels import linear

    def entry(code):
        def fn(v):
            v._obj.value = code
            return 0
        return staticmethod(fn)

    library = type("Library", (), {"oi_gemm_stream_status": entry(stream), "oi_gemm_few_status": entry(few)})
    monkeypatch.setattr(linear._lib, "load", lambda: library)
    assert linear.stream_status() == want and linear.few_status() == few


@pytest.mark.parametrize("design,name,streamed", [("rolevik", "A", True), ("luzitar", "A", True), ("bubalix", "A", False), ("delunex", "A", False)])
def test_steps_whose_experts_are_chosen_by_scores_run_with_streamed_products(monkeypatch, design, name, streamed):
    """Router scores: layers and head run under ``policy.streamed_products``, in that thread and for that long; a table of experts or
    no experts: they do not."""
    import importlib

    import torch

    from openinfer_b200.config.base import resolve_architecture
    from openinfer_b200.parts.model import Model
    raw = importlib.import_module(f"{design}_cases").CASES[name][0]
    entry = resolve_architecture(raw)
    model = Model(entry.build_spec(entry.config_cls.from_dict(raw)), torch.bfloat16)
    L = klib.load()
    seen = []

    def now(*_):
        was = L.oi_streamed_products(0)
        L.oi_streamed_products(was)
        seen.append(bool(was))
        return None, None

    model.native_step = False
    monkeypatch.setattr(model, "forward", now)
    monkeypatch.setattr(model, "logits", now)
    model.run(None, torch.zeros(1))
    now()
    assert model.routes_by_score == streamed and seen == [streamed, streamed, False]


@pytest.mark.parametrize("N,K,slices", [
    (4096, 4096, 8), (4224, 4096, 8), (4225, 4096, 4), (4224, 2048, 4),     # 256, 264, 272 CTAs in clusters of 8; short slices
    (6144, 4096, 4), (8960, 1024, 4), (8961, 1024, 2), (9216, 2048, 2),     # 192, 280, 284, 288 CTAs in clusters of 4
    (16384, 512, 2), (16512, 2048, 1), (16512, 3072, 2), (18816, 8192, 2),  # 256 and more in clusters of 2, short and long slices
    (18945, 8192, 1), (128, 64, 1), (128, 192, 1), (128, 256, 2), (128, 320, 2)])
def test_slices_of_the_streaming_product_run_at_once(N, K, slices):
    assert klib.load().oi_stream_slices(N, K) == slices
