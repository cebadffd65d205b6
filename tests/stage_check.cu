// stage_plan (csrc/tabstage.cuh) on the host: prints, for the profile type and the
// launch's step given, 1 for each table that is staged, in the order of StageTable.
#include <cstdio>
#include <cstdlib>

#include "tabstage.cuh"

int main(int argc, char **argv)
{
    if(argc < 3) return 2;
    bhcb::EnvDev e{};
    e.ssp_type = std::atoi(argv[1]);
    e.nssp = 31;
    e.has_seg = e.ssp_type == bhcb::SSP_CLINEAR || e.ssp_type == bhcb::SSP_CUBIC || e.ssp_type == bhcb::SSP_PCHIP;
    e.ntop = e.nbot = 2;
    e.nrr = 101;
    size_t off[bhcb::ST_COUNT];
    const size_t used = bhcb::stage_plan(e, std::atoi(argv[2]) != 0, bhcb::STAGE_DEFAULT_BYTES, off);
    for(int k = 0; k < bhcb::ST_COUNT; ++k) std::printf("%d", off[k] != (size_t)-1);
    std::printf(" %zu\n", used);
    return 0;
}
