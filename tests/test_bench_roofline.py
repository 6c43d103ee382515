"""bench.py's roofline record: the parts of stage 2 count as one kernel group with the bytes of its
algorithm, also where the list of large steps takes most of the time."""
import bench


def test_stage2_parts_are_one_group():
    timed = {"mask": (0.2, 1), "flux": (3.0, 1), "stage2_first": (2.0, 1), "stage2_iter": (4.0, 1),
             "erosion": (5.0, 1)}
    ms = bench.roofline_groups({k: v[0] for k, v in timed.items()})
    assert ms == {"mask": 0.2, "flux": 3.0, "stage2": 6.0, "erosion": 5.0}
    dom = max(ms, key=ms.get)
    bpc = bench.bytes_per_cell(3, True)
    assert set(ms) == set(bpc) and all(b > 0 for b in bpc.values())
    cells, peak = 1 << 20, 6545.6
    line = bench.roofline_line(dom, None, bpc[dom] * cells / 6e-3 / 1e9, peak, "measured", 3.0e8,
                               bpc[dom] * cells, 6e-3, timed, 1, None, 0.05, 329)
    assert line["kernel"] == "stage2" and line["traffic_over_alg"] > 0.0
    assert line["kernel_ms_per_step"]["stage2_iter"] == 4.0


def test_groups_without_stage2():
    assert bench.roofline_groups({"mask": 1.0}) == {"mask": 1.0}
