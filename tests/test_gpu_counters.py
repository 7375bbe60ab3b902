"""Work counters are left at zero by the launches that used them: more launches than the ring has slots, of every kernel
that takes one, on two streams, and each frame like the first."""
import pytest

pytestmark = pytest.mark.gpu


def test_more_launches_than_slots(cuda, native):
    import chaos_gb300 as cg
    torch = cuda
    w, h = 70, 50
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    orbit = cg.Orbit("0.0", "1.0", 128, 60)
    m = cg.Module("mandelbrot")
    bufs = [[torch.zeros(w * h, dtype=torch.int32, device="cuda:0") for _ in range(3)] +
            [torch.zeros((h, 128 * 16), dtype=torch.uint8, device="cuda:0")] for _ in streams]
    torch.cuda.synchronize()

    def frame(tier):
        return cg.FrameDesc(width=w, height=h, max_iterations=60, samples_per_pixel=1, sample_mode=cg.SAMPLES_CENTER,
                            tier=tier, arith=cg.ARITH_PARITY, fractal=cg.MANDELBROT, seed=0,
                            center_x=0.0 if tier == cg.TIER_PERTURB_F64 else -0.5, center_y=0.0, pixel_size=0.04)

    descs = [frame(t) for t in (cg.TIER_F32, cg.TIER_F64, cg.TIER_PERTURB_F64)]

    def launch(k):
        s, b = streams[k % 2], bufs[k % 2]
        for d, c in zip(descs[:2], b):
            cg.render_frame(d, cg.FrameOut(counts=c.data_ptr()), stream=s, sync=False)
        cg.render_frame_perturb(descs[2], orbit, cg.FrameOut(counts=b[2].data_ptr()), stream=s, sync=False)
        m.render_main(b[3].data_ptr(), 128 * 16, w, h, (-2.0, -1.0, 1.0, 1.0), 60, 2.0, 1, stream=s)

    launch(0)
    launch(1)
    torch.cuda.synchronize()
    first = [t.clone() for t in bufs[0]]
    for k in range(1100):  # 4400 launches
        for t in bufs[k % 2]:
            with torch.cuda.stream(streams[k % 2]):
                t.zero_()
        launch(k)
        if k % 50 == 0 or k > 1090:
            torch.cuda.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(first, bufs[k % 2])), k
