"""The default tile of every pass, over sizes and line counts: within the kernel's limits (shared memory, threads,
even FFT tiles, tensor-core CTAs) and with enough warps; what check_program refuses would refuse the launch."""
import ctypes

import pytest

from pypde_gb300 import _lib
import pypde_gb300.navier.fused as F

SIZES = [5, 9, 17, 33, 50, 65, 97, 129, 163, 193, 257, 289, 385, 433, 513, 700, 1025]


@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("fft", [True, False])
def test_every_default_tile_fits(split, fft):
    for prog in F.build_programs("CN", fft, split=split):
        for n in SIZES:
            m = int(1.5 * n)
            fft_n = m if fft and prog.has_dct else 0
            if fft_n and not F.fft_ok(m):
                continue
            lcap = ((m if prog.has_dct else n) + 1) | 1
            for lines in (1, 3, 40, 151, 153, 300, 305, 455, 457, 609, 900, 1300, 2307, 4000, 9000, 40000):
                tb, nt, wc, sd, dm = F._pick(prog, lines, lcap, fft_n, lines)
                P = F.launch_program(prog, (lcap, fft_n), tb, nt, wc, sd, dm,
                                     F._dense_tc(prog, lines, lcap, nt, fft_n, dm))
                assert 64 <= nt <= F._max_threads(prog, fft_n, dm) and nt % 32 == 0 and not dm
                assert not fft_n or tb % 2 == 0
                smem = _lib.smem_bytes(P) + ctypes.sizeof(_lib.PgxInstance) + 1024
                assert smem <= F.SMEM_PER_SM, (prog.name, n, lines, tb, nt)
                if any(P.ops[i].k & _lib.DENSE_TC for i in range(P.nops) if P.ops[i].code == _lib.OP["DENSE"]):
                    assert nt <= F.MAX_THREADS_DENSE
