"""The fused mode's choice between the tile kernel and the interpreter: deep
graphs of few events, whose layers are a barrier each, go to the interpreter
where the words are many, and both give the oracle's tallies."""
import numpy as np
import pytest

from mcscram_b200 import graph as G
from mcscram_b200 import synth
from mcscram_b200.graph import AND, OR, probability_threshold


def _deep(events, width, layers, fan=2, seed=0):
    """`width` chains of `layers` gates that each read the gate before and events, under one OR."""
    rng = np.random.default_rng(seed)
    inputs, count = [], []
    for level in range(layers):
        for k in range(width):
            below = [events + (level - 1) * width + k] if level else []
            inputs += below + [int(x) for x in rng.integers(0, events, fan - len(below))]
            count.append(fan)
    inputs += [events + (layers - 1) * width + k for k in range(width)]
    count.append(width)
    n = width * layers + 1
    return G.FlatGraph(be_pdag_idx=np.arange(2, 2 + events), be_event_idx=np.arange(events),
                       be_threshold=probability_threshold(rng.uniform(0.05, 0.9, events)),
                       gate_op=[int(x) for x in rng.choice([AND, OR], n - 1)] + [OR], gate_k=np.zeros(n),
                       gate_in_begin=np.concatenate([[0], np.cumsum(count)[:-1]]), gate_in_count=count,
                       gate_neg_count=np.zeros(n), inputs=inputs, tally_nodes=[events + n - 1])


@pytest.mark.gpu
@pytest.mark.parametrize("events,width,layers,words,tile", [
    (60, 1, 800, 2048, True), (60, 1, 800, 70001, False), (20, 1, 200, 262144, False), (20, 1, 200, 4097, True),
    (500, 1, 800, 70001, False), (1000, 4, 800, 70001, False), (200, 16, 20, 70001, True)])
def test_deep_graphs(capi, oracle_mod, gpu, events, width, layers, words, tile):
    g = _deep(events, width, layers)
    with capi.Engine(g, mode=capi.MODE_FUSED) as e:
        assert (e.fused_kernel(words)[0] > 0) == tile
        e.run(3, 2, 7, words)
        ones, total = e.tallies()
    assert total == 2 * words * 64
    assert np.array_equal(ones, oracle_mod.tallies(g, 3, 2, 7, words))


@pytest.mark.gpu
def test_trees_as_they_are_stay_with_the_tile_kernel(capi, gpu):
    for g in (synth.config1(), synth.small_tree(4)):
        with capi.Engine(g, mode=capi.MODE_FUSED) as e:
            assert all(e.fused_kernel(w)[0] > 0 for w in (1, 4096, 1 << 18, 1 << 32))
    with capi.Engine(synth.config1(), mode=capi.MODE_STRIP) as e:
        with pytest.raises(capi.McgError):
            e.fused_kernel(1)
