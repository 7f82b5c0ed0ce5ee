"""The bytes per item that the stage rooflines count, against the path-state arrays that the
two kernels at the ends of a sample read and write (16-byte arrays, but the 8-byte
generator and the 4-byte queue)."""

from lambda_b200 import STAGE_BYTES

SIZES = {"rng": 8, "queue": 4, "image": 12}


def _bytes(reads, writes):
    return sum(SIZES.get(name, 16) for name in reads.split() + writes.split())


def test_banking_a_sample_reads_its_last_ray_and_hit():
    ended = "film radiance lam hit_id ray_o ray_d throughput"  # bank_sample, whatever ended the sample
    assert STAGE_BYTES["raygen"] == _bytes(ended + " rng", "film radiance lam rng ray_o ray_d throughput queue")
    assert STAGE_BYTES["finish"] == _bytes(ended, "image")
