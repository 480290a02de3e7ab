"""The shared memory that a block of the smoother's tile form asks for
(tile_request in csrc/internal.h, compiled here for the host): never less than
it needs, never more than a block may have, for any number of tiles on devices
of few and many SMs; and one even share per block where the grid covers the
SMs."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get('CUDA_HOME', '/usr/local/cuda')
MAIN = '''
#include <cstdio>
#include "internal.h"
int main() {
  for (int sms : {1, 4, 152})
    for (int need : {8, 9000, 70000, kTileMaxBytes})
      for (long long tiles = 1; tiles < 40000; tiles += tiles < 20 ? 1 : tiles / 7)
        std::printf("%d %d %lld %zu\\n", sms, need, tiles, tile_request(need, (int)tiles, sms));
}
'''


def test_request_of_any_number_of_tiles(tmp_path):
    if not os.path.exists(os.path.join(CUDA, 'include', 'cuda_runtime.h')):
        pytest.skip('no CUDA headers')
    src, exe = tmp_path / 'm.cpp', tmp_path / 'm'
    src.write_text(MAIN)
    subprocess.check_call(['g++', '-std=c++17', '-I', os.path.join(CUDA, 'include'), '-I',
                           os.path.join(ROOT, 'bsam-in-matlab_gb300', 'csrc'), '-o', str(exe), str(src)])
    rows = [tuple(map(int, l.split())) for l in subprocess.check_output([str(exe)], text=True).splitlines()]
    assert len(rows) > 400 and max(t // s for s, _, t, _ in rows) > 10000
    for sms, need, tiles, got in rows:
        assert need <= got <= 200 * 1024, (sms, need, tiles, got)
        per = -(-tiles // sms)
        if 4 * tiles >= sms and per <= 8 and need <= 9000:
            assert per * (got + 2048) <= 224 * 1024 and (got == 200 * 1024 or (per + 1) * got > 200 * 1024 // 2)
