// psg_ns3d_f64.cu -- FP64 3D engine of one grid size, PSG_GRID (compiled once per size, so that
// the sizes build in parallel).
#include "psg_ns3d_impl.cuh"
template <>
psg::Engine3DBase* psg::make_engine3d<double, PSG_GRID>() { return new psg::Engine3D<double, PSG_GRID>(); }
