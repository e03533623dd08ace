"""How a prompt is cut into passes of the many-row path: every row once, in order, slab boundaries at multiples of 16,
no pass beyond the workspace bound and no short one behind a whole one."""
from bitmtp_b200.model import PREFILL_CHUNK, PREFILL_TAIL, PREFILL_WAVE, prompt_waves


def test_prompt_waves_cover_the_prompt():
    for seq in [1, 15, 16, 17, 255, 256, 1023, 1024, 1025, 1279, 1280, 1281, 2048, 2303, 2304, 2900, 4096, 65536 + 3]:
        waves = prompt_waves(seq)
        assert [c0 for c0, _ in waves] == [sum(n for _, n in waves[:i]) for i in range(len(waves))]
        assert sum(n for _, n in waves) == seq
        assert all(c0 % PREFILL_CHUNK == 0 for c0, _ in waves)
        assert all(n == PREFILL_WAVE for _, n in waves[:-1]) and waves[-1][1] < PREFILL_WAVE + PREFILL_TAIL
        assert len(waves) == 1 or waves[-1][1] >= PREFILL_TAIL
