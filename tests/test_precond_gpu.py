

def test_cycles_are_not_collected_while_a_graph_is_captured():
    """Destroying a captured graph invalidates any capture under way; a cycle may hold one."""
    import gc

    from heavyball_b200.utils import core

    def cycle_with_a_graph():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            torch.ones(8, device="cuda")
        holder = [graph]
        holder.append(holder)

    gc.collect()
    threshold = gc.get_threshold()
    cycle_with_a_graph()
    fresh = torch.cuda.CUDAGraph()
    try:
        gc.set_threshold(1, 1, 1)
        with core._captured_into(fresh):
            objects = [[i] for i in range(2000)]  # would set off a collection of every generation
            x = torch.ones(8, device="cuda") * 3
    finally:
        gc.set_threshold(*threshold)
    assert gc.isenabled() and len(objects) == 2000
    fresh.replay()
    assert x.tolist() == [3.0] * 8
