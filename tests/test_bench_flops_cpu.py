"""The FP32 operations that the bench line charges a mixed line sum are those that the committed
counters show, in both counted windows (their figures have three or four digits: 0.5 %)."""
import re
import sys

from conftest import ROOT

sys.path.insert(0, str(ROOT))


def test_line_sum_flops_match_the_counters():
    import bench
    text = (ROOT / "profiles" / "linesum_iasi400k.txt").read_text()
    kernels = re.findall(r"core_pairs (\S+), evaluated_pairs (\S+)\nfw_tree\S+ .*? FP32 (\S+) .*?\nfw_leaf\S+ .*? FP32 (\S+) ", text)
    assert len(kernels) == 2
    for core, evaluated, tree, leaf in kernels:
        counted = float(tree) + float(leaf)
        assert abs(bench.line_sum_flops(float(evaluated), float(core)) - counted) <= 5e-3 * counted
