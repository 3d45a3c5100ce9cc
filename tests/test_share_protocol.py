"""The work sharing between warps (csrc/share.cuh) on the host: its own code, compiled against a
model of the device (tests/cpp/model_kernels.h) in which every memory operation is a step, under
random schedules with blocks that start late.  Every handed-on task runs, once, and none stays in the
queue for the next launch; with long waits, and with waits so short that many run out."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def build(tmp_path, polls):
    src = open(os.path.join(ROOT, 'rtcollisiondetection_b200', 'csrc', 'share.cuh')).read()
    # volatile accesses become steps of the model, the block's shared word its LiveWord
    src = re.sub(r'(?:const )?volatile uint32_t\* s_live', 'LiveWord* s_live', src)
    src, n = re.subn(r'\*\((?:const )?volatile ([a-z0-9_ ]+)\*\)', r'*(model::Step<\1>)', src)
    assert n >= 4
    src, n = re.subn(r'kSharePolls = 1 << 16', 'kSharePolls = %d' % polls, src)
    assert n == 1
    (tmp_path / 'share.cuh').write_text(src)
    cpp = os.path.join(ROOT, 'tests', 'cpp')
    shutil.copy(os.path.join(cpp, 'model_kernels.h'), tmp_path / 'kernels.h')
    exe = str(tmp_path / 'share_model')
    cxx = shutil.which('g++') or shutil.which('c++')
    subprocess.check_call([cxx, '-std=c++17', '-O1', '-I', str(tmp_path), os.path.join(cpp, 'share_model.cpp'), '-o', exe])
    return exe


@pytest.mark.parametrize('polls', [1 << 16, 30])
def test_every_task_runs_once(tmp_path, polls):
    out = subprocess.run([build(tmp_path, polls), '3000', '7'], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
