"""What the host does with the word that a kernel raises when one of its bounded waits has run out. The word is set from the
host (tests/cpp/error_word.cu reaches it); no wait runs out on the GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import vkllama_b200 as vk
from oracle import oracle as O
from vkllama_b200 import build as B

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def words(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("words") / "error_word.so")
    subprocess.check_call([B.NVCC] + B.FLAGS + ["-shared", "-I", B.CSRC, os.path.join(ROOT, "tests", "cpp", "error_word.cu"), "-o", so])
    L = C.CDLL(so)
    L.raise_model_word.argtypes = [C.c_void_p]
    return L


def test_block_forward_reports_its_own_waits(dev, words):
    """Rows of a block whose projections gave up are not handed out as a success, and the next call is not blamed."""
    dm = vk.Model(dev, 128, 2, 256, 100, 1, 64)
    dm.synth_weights(71)
    x = O.synth_f16(71, 5, 20 * 128).reshape(20, 128)
    want = dm.block_forward(0, x, 0)
    assert words.raise_model_word(dm.h) == 0
    with pytest.raises(vk.VklError) as e:
        dm.block_forward(0, x, 0)
    assert e.value.code == 13
    assert (dm.block_forward(0, x, 0) == want).all()
    dm(np.arange(12, dtype=np.uint32), 0)
    dm.close()
