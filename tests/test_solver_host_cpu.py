"""Host-side decision logic of the solvers, without a GPU: the sweep autotuner's choice."""
from edge_to_b200.solvers import CuMultiGrid, pick_sweep_pattern


def _retime(table, fail=()):
    def f(pattern):
        key = tuple(pattern)
        return table[key], key not in fail, 0
    return f


def test_sweep_choice_tie_goes_to_fewer_sweeps():
    m = CuMultiGrid.SWEEP_MARGIN
    # the fastest is also the cheapest: kept
    runs = [[85.2, [1, 1, 1, 1, 1], 195], [88.7, [1, 2, 2, 2, 2], 147], [99.5, [2, 2, 2, 2, 2], 149]]
    best = pick_sweep_pattern(runs, _retime({(1, 1, 1, 1, 1): 85.0}), m)
    assert best[1] == [1, 1, 1, 1, 1] and best[0] == 170.2
    # more sweeps 3 % faster on both timings: within the margin, the cheapest is kept
    runs = [[100.0, [1, 1, 1], 10], [97.0, [1, 2, 2], 8]]
    best = pick_sweep_pattern(runs, _retime({(1, 1, 1): 100.0, (1, 2, 2): 97.0}), m)
    assert best[1] == [1, 1, 1]
    # 20 % faster: the pattern with more sweeps wins
    runs = [[100.0, [1, 1, 1], 10], [80.0, [1, 2, 2], 8]]
    best = pick_sweep_pattern(runs, _retime({(1, 1, 1): 100.0, (1, 2, 2): 80.0}), m)
    assert best[1] == [1, 2, 2] and best[0] == 160.0
    # the fastest fails to converge when timed again: the cheapest is kept
    runs = [[100.0, [1, 1, 1], 10], [60.0, [2, 2, 2], 8]]
    best = pick_sweep_pattern(runs, _retime({(1, 1, 1): 100.0, (2, 2, 2): 60.0}, fail={(2, 2, 2)}), m)
    assert best[1] == [1, 1, 1]
    # the input list is not modified
    assert runs[0][0] == 100.0


def test_sweep_choice_falls_back_when_no_contender_converges_again():
    m = CuMultiGrid.SWEEP_MARGIN
    fallback = [3, 3, 3]
    # the only contender (fastest = cheapest) fails on its retime
    runs = [[100.0, [1, 1, 1], 10], [120.0, [2, 2, 2], 8]]
    best = pick_sweep_pattern(runs, _retime({(1, 1, 1): 100.0}, fail={(1, 1, 1)}), m, fallback=fallback)
    assert best == (0.0, [3, 3, 3], 0)
    # both contenders fail on their retimes
    runs = [[100.0, [1, 1, 1], 10], [60.0, [2, 2, 2], 8]]
    best = pick_sweep_pattern(runs, _retime({(1, 1, 1): 100.0, (2, 2, 2): 60.0}, fail={(1, 1, 1), (2, 2, 2)}), m,
                              fallback=fallback)
    assert best == (0.0, [3, 3, 3], 0)


def test_row_plan_of_the_one_launch_product_is_made_with_the_problem():
    """The search for the rows per block tries up to 4,096 splits on the host: it runs at a problem's
    creation, and the launch itself holds no loop."""
    import os
    import re
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "edge_to_b200", "csrc")
    solver, fields = (open(os.path.join(csrc, f)).read() for f in ("solver.cu", "fields.cu"))
    calls = [m.start() for m in re.finditer(r"user3_rows\(", solver)]
    create = solver.index("\nint edge_problem_create(")
    assert len(calls) == 1 and create < calls[0] < solver.index("\n}\n", create)
    launch = fields[fields.index("static int user3_launch("):]
    launch = launch[:launch.index("\n}\n")]
    assert "<<<" in launch and "for (" not in launch and "user3_rows" not in launch and "user3_chunk" not in launch


def test_the_one_launch_cycle_is_loaded_without_the_batched_solve():
    """A process loads all kernels of a translation unit at its first launch from it: the one-launch 2-D
    cycle, which every small 2-D solve uses, stays apart from the 33 kernels of the batched solve (60 ms
    of a process's first solve)."""
    import os
    from edge_to_b200 import build
    units = {s: open(os.path.join(build.CSRC, s)).read() for s in build.SOURCES}
    cycle = [s for s, t in units.items() if "k_vtail2<" in t]
    batch = [s for s, t in units.items() if "k_batch_pcg<" in t]
    assert len(cycle) == len(batch) == 1 and cycle != batch
