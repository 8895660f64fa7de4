// An upper yield limit below -1, whose square exceeds 1, under a lower one: every singular value of
// an F near a rotation is above the upper limit and ends at the lower one, as FP64 clamps.
// precompute<float, float> and <float, double>
// against the FP64 update on the same FP32 inputs. Per precision, in units of 2^-24, a NaN
// kept: the largest difference of Fe and Re, and of Jp and Je (relative).
#include "mpm_math.cuh"
#include <cmath>
#include <cstdio>
#include <random>

using namespace mpm;

static void worst(double& a,double b){if(!(b<=a)) a=b;}

template<class TS> static void check(const char* name)
{
    std::mt19937_64 g(3);
    std::uniform_real_distribution<double> u(-1.,1.);
    const float cy=.5f,sy=-2.f;
    double entries=0,scalars=0;
    for(int it=0;it<4000;++it){
        const double a=3.2*u(g),c=std::cos(a),s=std::sin(a),e=.006*u(g);
        float Fm[9]={(float)(c*(1+e)),(float)-s,0.f,(float)(s*(1+e)),(float)c,0.f,0.f,0.f,(float)(1-e)},Rm[9],lam,mu,Je,Jp=1.f;
        double Fx[9],Rx[9],lx,mx,Jx,Jq=1.;
        for(int k=0;k<9;++k) Fx[k]=Fm[k];
        precompute<float,TS>(Fm,Jp,1e4f,2e4f,1,0.f,cy,sy,10.f,Rm,lam,mu,Je);
        precompute<double,double>(Fx,Jq,1e4,2e4,1,0.,(double)cy,(double)sy,10.,Rx,lx,mx,Jx);
        for(int k=0;k<9;++k){worst(entries,std::fabs(Fm[k]-Fx[k]));worst(entries,std::fabs(Rm[k]-Rx[k]));}
        worst(scalars,std::fabs(Jp-Jq)/std::fabs(Jq));worst(scalars,std::fabs(Je-Jx)/std::fabs(Jx));}
    std::printf("%s_entries %.4f %s_scalars %.4f ",name,entries*std::ldexp(1.,24),name,scalars*std::ldexp(1.,24));
}
int main()
{
    check<float>("fp32");check<double>("mixed");
    std::printf("\n");
    return 0;
}
