"""Traffic figures that the bench publishes (profiles/roofline_traffic.json): each
names a kernel that the sources define and a summary that is there and has the
figure's launch.  Needs no GPU."""
import glob
import json
import os
import re

from mnpbem_b200.build import CSRC, ROOT


def test_traffic_figures_are_of_present_kernels():
    src = ''.join(open(f).read() for f in glob.glob(os.path.join(CSRC, '*.cu*')))
    with open(os.path.join(ROOT, 'profiles', 'roofline_traffic.json')) as f:
        table = json.load(f)
    assert table
    for cls, t in table.items():
        name = re.match(r'\w+', t['launch']).group(0)
        assert re.search(r'\b%s\(' % name, src), (cls, name)
        with open(os.path.join(ROOT, t['source'])) as f:
            assert name in f.read(), (cls, t['source'])
        assert 0 < t['algorithmic_bytes'] < 1.5 * t['dram_bytes']
