"""Shared memory of cluster kernels that allocate tensor memory: those that share an SM must not ask for more than its 512 columns together, or CTAs
of two clusters on two streams can wait for each other for good."""
import ctypes as C

SM_BYTES, SYSTEM_BYTES, LEAST_STAGES = 228 * 1024, 1024, 2 * (128 + 16) * 128      # the smallest ring of a clustered product: two stages, 16 rows


def test_pairs_leave_no_room_for_a_second_allocation(lib):
    """A pair's CTA has all 512 columns, so no other CTA of a cluster may fit beside it: not the smallest there is today, nor one with the least
    shared memory that 32 columns come with."""
    smem, pairs = C.c_int32(0), 0
    for M in (256, 1000, 2048, 2500, 3333, 4096, 8192):
        for N, K in ((16, 64), (2048, 2048), (2048, 4096), (12288, 2048), (12352, 2048)):
            form = lib.kb2_linear_bf16_form(M, N, K, 0, C.byref(smem))
            if form <= 0:
                assert smem.value == 0
                continue
            pairs += 1
            assert 96 <= form <= 256 and form % 16 == 0
            assert smem.value >= 430 * 512 - SYSTEM_BYTES
            left = SM_BYTES - (smem.value + SYSTEM_BYTES)
            assert left < LEAST_STAGES + SYSTEM_BYTES and left < 430 * 32
    assert pairs > 10
