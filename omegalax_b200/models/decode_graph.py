"""Single-token steps as recorded CUDA graphs.

A decode step launches a few small kernels per layer, so its time is launch overhead unless it is
recorded once and replayed.  A step's shapes depend on the cache only (one row per sequence, idle rows
marked), so the recording lives on the cache: the first single-token step runs eagerly, the second one
records, later ones copy their token batch into the recorded buffers and replay.
"""
from __future__ import annotations

import os
import threading

import torch

from ..ops import kernels as K
from ..ops import lib


# A recording that leaves less than this to the device gives the allocator's free memory back first: while one is made
# the allocator cannot do so, and a step's temporaries come from memory of its own.
_SPARE = 1 << 30


def other_threads() -> bool:
    return threading.active_count() > 1


class DecodeGraph:
    def __init__(self, model, cache, batch):
        self.batch = batch            # the recorded step reads these tensors
        before = K.launch_count()
        self.graph = torch.cuda.CUDAGraph()
        # ``torch.cuda.graph`` would wait for the device and give the allocator's free memory back first, to be asked for
        # again: the second step of a fresh cache took 9.0 ms so and takes 5.1 (8 layers of 4096 channels; 3.1 call by call, 1.6 recorded)
        if torch.cuda.mem_get_info()[0] < _SPARE:
            torch.cuda.empty_cache()
        here, side = torch.cuda.current_stream(), torch.cuda.Stream()
        side.wait_stream(here)
        with torch.cuda.stream(side):
            # other threads go on allocating while this one records
            self.graph.capture_begin(capture_error_mode="thread_local")
            try:
                # no kernel of a step writes parameters, so products may read theirs ahead of the kernel before them
                lib.call("ob_overlap_launches", 1)
                self.out = model.run_layers(batch, cache)
            finally:
                lib.call("ob_overlap_launches", 0)
                self.graph.capture_end()
        here.wait_stream(side)
        self.launches = K.launch_count() - before
        self.model = model
        self.every = False            # the last call had a token for every sequence, as far as the model says so
        self.asked, self.arrived = None, torch.cuda.Event()     # what a step that runs ahead asks the device for (pinned)

    @staticmethod
    def enabled() -> bool:
        return os.environ.get("OMEGALAX_B200_DECODE_GRAPH", "1") == "1"

    @staticmethod
    def recorded(model, cache, key) -> "DecodeGraph | None":
        """The recording that a step with this key would replay."""
        state = cache.decode_graph
        if state is None or state[0] is not model or state[1] is None or state[2] != key or not DecodeGraph.enabled():
            return None
        return state[1]

    def replay(self):
        K.add_launches(self.launches)
        self.graph.replay()
        return self.out

    @staticmethod
    def step(model, cache, batch, key=None, alone: bool = False):
        """Residual rows of a single-token batch; the tensor is reused by the next step.  A recording serves while
        ``key`` (what the model runs and where its weights lie) compares equal.  With ``alone`` nothing is recorded while the
        program has other threads: one that waits for the device or draws random numbers there meanwhile would be
        refused.  Replays disturb nobody."""
        state = cache.decode_graph
        if not DecodeGraph.enabled():
            return model.run_layers(batch, cache)
        if state is None or state[0] is not model or state[2] != key:
            cache.decode_graph = (model, None, key)
            return model.run_layers(batch, cache)
        graph = state[1]
        if graph is None:
            if alone and other_threads():
                return model.run_layers(batch, cache)
            graph = DecodeGraph(model, cache, batch)
            cache.decode_graph = (model, graph, key)
            graph.graph.replay()
            return graph.out
        graph.batch.flat.copy_(batch.flat)
        return graph.replay()
