"""Host-side rules of the training backward."""
import pytest

WAVE = 304 * 128


@pytest.mark.parametrize("chunk", [128, 640, 86 * 128, WAVE, 4 * WAVE, 5 * WAVE, 36 * WAVE, 60 * WAVE])
@pytest.mark.parametrize("n", [0, 1, 128, 40000, 1260000, 1400000, 1400833, 1700000, 2090000,
                               2150000, 9000000])
def test_chains_of_weight_gradients_end_at_their_limit(n, chunk):
    """Additions of the longest FP32 chain of layers 2 and 3: a block (of 76)
    takes equal runs of a chunk's 128-sample tiles, one chain for every other
    sample, and the chains go on over nsvf_field_train_chain_chunks chunks.
    At most 9,216, or what one chunk holds; and no more sets of chains than
    that asks for."""
    from nsvf_gb300._lib import LIB
    group = LIB.nsvf_field_train_chain_chunks(n, chunk)
    assert group >= 1
    chunks = [min(chunk, n - a) for a in range(0, n, chunk)]
    per = [-(-(-(-c // 128)) // 76) * 64 for c in chunks]
    for k in range(0, len(chunks), group):
        assert sum(per[k:k + group]) <= max(9216, per[0])
    sets, most = -(-len(chunks) // group), max(1, 9216 // per[0]) if per else 1
    assert sets == -(-len(chunks) // most)


def test_chain_chunks_rejects_what_the_backward_does():
    from nsvf_gb300._lib import LIB
    assert LIB.nsvf_field_train_chain_chunks(-1, 128) == -1
    assert LIB.nsvf_field_train_chain_chunks(5, 0) == -1


@pytest.mark.parametrize("ns,rays,chunk_rays,want", [
    (0, 0, 1024, 128), (1, 1, 1, 128), (1000, 10, 1, 128), (1300, 10, 1, 256),
    (WAVE // 2 * 8, 8, 1, WAVE), (WAVE // 2 * 8 - 8, 8, 1, WAVE // 2),
    (340000, 2048, 64, 84 * 128), (1400000, 8192, 1024, 4 * WAVE), (1400000, 8192, 8192, 36 * WAVE)])
def test_backward_chunk_follows_chunk_rays(ns, rays, chunk_rays, want):
    """A caller who lowers chunk_rays gets a chunk, and a workspace, as much
    smaller; from half a wave of the GPU on the chunk is whole waves."""
    from nsvf_gb300 import train
    from nsvf_gb300._lib import LIB
    chunk = train.chunk_samples(ns, rays, chunk_rays)
    assert chunk == want
    n = ns * chunk_rays / max(rays, 1)
    assert chunk <= max(2 * n, n + 128)
    fixed = LIB.nsvf_field_train_backward_floats(0, 128)
    assert LIB.nsvf_field_train_backward_floats(ns, chunk) - fixed <= 1100 * min(chunk, ns + 128)
