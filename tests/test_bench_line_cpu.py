"""The benchmark prints one line that a caller with a few KB of buffer keeps whole; every block's full record
goes elsewhere."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def test_the_line_is_short_and_complete():
    import bench
    kern = {k: {'ms_per_launch_live': 0.03, 'share': 0.4, 'launches_per_solve': 1500} for k in ('k_stage_op', 'k_limit_dot')}
    roof = {'bound': 'hbm', 'kernel': 'k_stage_op', 'achieved': 1000.0, 'peak': 6787.2, 'unit': 'GB/s', 'frac': 0.147,
            'traffic': 58.5e6, 'note': 'n' * 2000, 'fp64_rate': {'kernels': kern}}
    side = {'value': 5.0e10, 'kernels': kern, 'roofline': roof, 'launch': {'flags': 0}}
    result = {k: 1.25 for k in bench.HEADLINE}
    result.update(config={'model': 'm' * 200, 'launch': {'flags': 0}}, clocks={'sm_mhz': 2000, 'reasons': []},
                  e2e={'value': 1e10, 'unit': 'u', 'h2d_bytes_per_step': 1, 'd2h_bytes_per_step': 1, 'timing': 't' * 200},
                  roofline=roof, kernels=kern, whole_stage={'frac': 0.2}, metric_note='x' * 500, fp32=side, df32=side,
                  adjoint={p: {m: {'backward_over_forward': 2.5, 'backward_ms': 1.0} for m in ('stored', 'snapshots_20')}
                           for p in ('fp64', 'fp32')},
                  large={p: side for p in ('fp32', 'fp32_volume_mma', 'fp64')},
                  ensemble=dict(side, groups={1: side, 2: side}))
    line = bench.headline(result)
    assert all(k in line for k in bench.HEADLINE)
    assert line['value'] == result['value'] and line['e2e'] == result['e2e']
    assert line['side']['fp32'] == 5.0e10 and line['side']['large.fp64'] == 5.0e10
    assert line['side']['ensemble.groups.1'] == 5.0e10
    assert line['side']['adjoint.fp32.snapshots_20'] == 2.5
    assert len(json.dumps(line)) < 4000 < len(json.dumps(result))


def test_the_rates_divide_the_present_kernels_counters():
    """FP64 operations and DRAM bytes per launch are constants: they have to be the ones of the counter
    summary of the kernels in the tree, not of kernels that these replaced."""
    import bench
    path = os.path.join(os.path.dirname(bench.__file__), 'profiles', 'stage_kernels_131k_fp64_full.md')
    present = open(path).read().split('## The FP64 forms before')[0]
    row = {r[1].strip(): [c.strip() for c in r[2:-1]] for r in (x.split('|') for x in present.splitlines()) if len(r) == 6}
    names = ('k_stage_op', 'k_limit_dot', 'k_limit')
    per = [[float(x) for x in row[k + ' / element']] for k in ('DFMA', 'DADD', 'DMUL')]
    for i, name in enumerate(names):
        flops = bench.MEASURED_FP64_FLOPS[('gauss_slot_131k_p2', name)]
        assert flops == float(row['FP64 flops / element (2 DFMA + DADD + DMUL)'][i])
        assert abs(flops - (2 * per[0][i] + per[1][i] + per[2][i])) <= 0.25      # four roundings of 0.05
        assert bench.MEASURED_TRAFFIC[('gauss_slot_131k_p2', 'fp64', name)] == float(row['DRAM read + write (MB)'][i]) * 1e6
