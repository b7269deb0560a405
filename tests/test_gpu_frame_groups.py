"""GPU: a batch of frames is split into groups that decode side by side; every
count of groups and group sizes (one frame each, uneven ones, a batch past the
limit that stays one group) gives each frame the outputs it has alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [2, 8, 9, 17, 64, 65])
def test_groups_match_frames_alone(gpu_ctx, count):
    from dvc_b200 import bitstream as bs, decoder, encoder, synth
    kinds = []
    for q in (1, 4, 8):  # mixed step lists within and between groups
        ori, key = synth.make_sequence("qcif", 3, 30 + q)
        st = bs.parse_wz(encoder.encode_sequence(ori, 2, q))
        kinds.append((st, st.frames[1], key))

    def item(i):
        st, fr, key = kinds[i % 3]
        return decoder.frame_item(st, fr, np.array(key, np.uint8))

    alone = [gpu_ctx.decode_wz_frames([item(i)])[0] for i in range(3)]
    for i, out in enumerate(gpu_ctx.decode_wz_frames([item(i) for i in range(count)])):
        want = alone[i % 3]
        assert np.array_equal(out["recon"], want["recon"]), i
        assert out["wz_bits"] == want["wz_bits"], i
        assert np.array_equal(out["planes"][:, :3], want["planes"][:, :3]), i
        assert np.array_equal(np.asarray(out["entropy"]).view(np.uint32), np.asarray(want["entropy"]).view(np.uint32)), i
