"""Model of what the copying thread of the layer kernel (csrc/s14_moe_umma.cu) leaves in flight when a role gives up, run on the CPU.

Units go into the ring's slots in turn, a phase of the slot's barrier each; a layer's router rows, asked for once the layer before has its
routes, are a phase of a barrier of their own.  The thread may stop anywhere.  At the end it waits for the last phase of the slots that the
last `ring` units went to, and for the last phase of the rows.  Property: nothing is in flight then."""
import random

import pytest


def in_flight(rng, wait_for_rows):
    """One random run: the phases of each barrier that were armed and that nobody has waited for when the CTA leaves."""
    ring, layers, units_per_layer = 2 * rng.randrange(1, 7), rng.randrange(1, 6), rng.randrange(1, 30)
    armed, units, rows, stop = set(), 0, 1, rng.randrange(0, 150)
    armed.add(("rows", 0))
    for layer in range(layers):
        if layer:   # the roles have waited for this layer's rows, or the thread does not come here
            armed.discard(("rows", layer - 1))
        for unit in range(units_per_layer):
            if units >= stop:
                break
            slot, phase = units % ring, units // ring
            if phase:   # a slot is filled again when its MMAs, which waited for the copy, are done
                armed.discard((slot, phase - 1))
            armed.add((slot, phase))
            units += 1
            if unit == 0 and layer + 1 < layers:
                armed.discard(("rows", layer))
                armed.add(("rows", layer + 1))
                rows = layer + 2
    for u in range(max(0, units - ring), units):
        armed.discard((u % ring, u // ring))
    if wait_for_rows:
        armed.discard(("rows", rows - 1))
    return armed


@pytest.mark.parametrize("wait_for_rows", [True, False])
def test_nothing_is_in_flight_when_a_cta_leaves(wait_for_rows):
    rng = random.Random(3)
    assert any(in_flight(rng, wait_for_rows) for _ in range(5000)) != wait_for_rows
