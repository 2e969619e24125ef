"""The memory of the access tables goes back to the device when the last structure is gone, up to the stock that small structures are
built from (256 MiB).  In a process of its own, where no other test keeps a structure alive."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import torch, pyapr
from pyapr import synthetic
torch.cuda.init()
image = synthetic.blob_image((256, 512, 512), 625, 3, device="cuda")
arrays = synthetic.apr_from_image(image)
del image
small = pyapr.apr_from_arrays(arrays); small.init_cuda(); small.plan(2); del small          # kernels and libraries are loaded
torch.cuda.synchronize(); torch.cuda.empty_cache()
before = torch.cuda.mem_get_info()[0]
apr = pyapr.apr_from_arrays(arrays)
apr.init_cuda()
for dl in range(4):
    apr.plan(dl)
used = apr.cuda_device_bytes()
del apr
torch.cuda.synchronize(); torch.cuda.empty_cache()
kept = before - torch.cuda.mem_get_info()[0]
print(used >> 20, kept >> 20)
assert used > 600 << 20 and kept <= 320 << 20, (used, kept)
"""


def test_tables_go_back_with_the_last_structure():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "apr-cnn_b200"))
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
